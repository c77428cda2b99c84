"""The tensor-core Kubo sums where a fill of 16 records, a tile of 128 frequencies or a tile of 104 columns
is ragged: records left over in the last fill of a k-point (num_wann 4 to 9), k-points without records, one
frequency, one more than a tile, one and several column tiles.  Against the CUDA-core product of the same
records: both sum FP32 factors (relative error a few 2^-24, two roundings apart) of at most num_wann^2 records."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import autotune, models, system as wsys  # noqa: E402
import wbgpu  # noqa: E402

C = wbgpu.calculators


@pytest.mark.parametrize('nw,nE,nO,nk', [(4, 1, 1, (1, 1, 1)), (5, 2, 127, (3, 2, 1)), (7, 12, 128, (5, 2, 2)),
                                         (9, 4, 129, (4, 3, 3)), (6, 13, 257, (9, 6, 5))])
def test_ragged_fills(nw, nE, nO, nk):
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, np.diag([3.0, 3.5, 4.0]), seed=nw))
    EF = np.linspace(-40.0, 1.0, nE) if nE > 1 else np.array([0.2])  # the lowest: no records at any k-point
    om = np.linspace(0.0, 3.0, nO)
    p = dict(Efermi=EF, omega=om, smr_fixed_width=0.3)
    cal = {'opt': C.OpticalConductivity(**p), 'opt_G': C.OpticalConductivity(smr_type='Gaussian', **p),
           'shift': C.ShiftCurrent(sc_eta=0.1, **p), 'inj': C.InjectionCurrent(**p)}
    res = []
    for engine in (1, 2):
        autotune.set_value(autotune.KUBO_ENGINE, 1, 0, engine)
        try:
            res.append(wbgpu.run(s, wbgpu.Grid(s, NKdiv=1, NKFFT=nk), cal, precision='mixed'))
        finally:
            autotune.set_value(autotune.KUBO_ENGINE, 1, 0, 0)
    for q in cal:
        a, b = res[0][q].data, res[1][q].data
        assert np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(b)), q
