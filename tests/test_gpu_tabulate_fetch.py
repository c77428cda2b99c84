"""The tabulated values come back whole, whichever columns are asked for and however many rows there are: cut on
the host below 4 096 rows, packed on the device from there on, one batch or several."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import models, system as wsys  # noqa: E402
import wbgpu  # noqa: E402

T = importlib.import_module('wbgpu.tabulate')
R = importlib.import_module('wbgpu.run')


@pytest.mark.parametrize("nw,fft", [(4, (1, 1, 1)), (5, (7, 9, 13)), (4, (8, 8, 16)), (5, (9, 9, 11))])
def test_columns_and_sizes(nw, fft, monkeypatch):
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, np.diag([3.0, 3.5, 4.0]), seed=nw))
    grid = wbgpu.Grid(s, NKdiv=2, NKFFT=fft)
    every = wbgpu.tabulate(s, grid, T.QUANTITIES)
    for q in T.QUANTITIES:  # the same kernels: the same bits
        one = wbgpu.tabulate(s, grid, (q,))
        assert np.array_equal(one[q], every[q]) and np.isfinite(one[q]).all(), q
        assert one[q].shape == (grid.nk_per_block * 8, nw) + (() if q == 'energy' else (3,))
    monkeypatch.setattr(R, 'choose_batch', lambda *a: 3)  # batches of 3, 3 and 2 blocks
    few = wbgpu.tabulate(s, grid, ('energy', 'band_gradients'))
    assert np.allclose(few['energy'], every['energy'], rtol=0, atol=1e-12)
