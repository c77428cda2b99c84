"""FP64 results are the same bits however the blocks of a run are batched."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import models, system as wsys  # noqa: E402
import wbgpu  # noqa: E402

C = wbgpu.calculators
LAT = np.diag([3.0, 3.5, 4.0])


def _same(s, grid, calculators, batches):
    ref = wbgpu.run(s, grid, calculators(), blocks_per_batch=batches[0])
    for nb in batches[1:]:
        got = wbgpu.run(s, grid, calculators(), blocks_per_batch=nb)
        for q in ref:
            assert np.isfinite(ref[q].data).all() and np.abs(ref[q].data).max() > 0, q
            assert np.array_equal(got[q].data, ref[q].data), (q, nb)


@pytest.mark.parametrize("nw,nEF,nomega", [(4, 1, 5), (9, 5, 61), (12, 3, 130)])
def test_frequency_sums(nw, nEF, nomega):
    """Every kind of FP64 frequency sum (real or complex factors and elements), one block of 64 k-points at a time
    and in larger batches."""
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, LAT, seed=nw, keys=('Ham', 'AA', 'SS')))
    opt = dict(Efermi=np.linspace(-0.5, 0.5, nEF) if nEF > 1 else np.array([0.0]), omega=np.linspace(0.0, 4.0, nomega),
               smr_fixed_width=0.05)
    cal = lambda: {'optical': C.OpticalConductivity(**opt), 'shift': C.ShiftCurrent(sc_eta=0.04, **opt),
                   'injection': C.InjectionCurrent(**opt), 'shc': C.SHC(SHC_type='simple', **opt)}
    _same(s, wbgpu.Grid(s, NKdiv=3, NKFFT=(4, 4, 4)), cal, (1, 5, 27))
