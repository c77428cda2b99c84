"""The scans' launch shapes: lanes a k-point, k-points a block and blocks an SM follow from the sizes, and the
fixed-point sums make the result the same bits in every shape.  One block of 512 k-points at a time (the smallest
shape) against all 13 824 at once (the largest), at the edges of the lane counts, few and many levels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import models, system as wsys  # noqa: E402
import wbgpu  # noqa: E402

C = wbgpu.calculators


@pytest.mark.parametrize("nw,nEF,precision", [(3, 5, 'mixed'), (8, 501, 'mixed'), (9, 1001, 'mixed'), (16, 3000, 'mixed'),
                                              (17, 11, 'mixed'), (33, 201, 'mixed'), (4, 101, 'fp64'),
                                              (17, 1001, 'fp64')])
def test_same_bits_in_every_shape(nw, nEF, precision):
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, np.diag([3.0, 3.5, 4.0]), seed=nw))
    EF = np.linspace(-2.0, 2.0, nEF)
    cal = {'ahc': C.AHC(Efermi=EF), 'ohmic': C.Ohmic_FermiSurf(Efermi=EF), 'dos': C.DOS(Efermi=EF)}
    if precision == 'fp64':
        cal['dipole'] = C.BerryDipole_FermiSurf(Efermi=EF)
    grid = wbgpu.Grid(s, NKdiv=3, NKFFT=(8, 8, 8))
    run = lambda nb: wbgpu.run(s, grid, cal, precision=precision, blocks_per_batch=nb)
    a, b = run(1), run(27)
    for q in cal:
        assert np.isfinite(a[q].data).all() and np.abs(a[q].data).max() > 0, q
        assert np.array_equal(a[q].data, b[q].data), q
