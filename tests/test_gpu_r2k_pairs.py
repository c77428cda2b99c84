"""R -> k transform on conjugate pairs of R components: symmetric, one-sided and ragged R sets against the
direct sum, and the FP64 path's lower triangles."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
import wbgpu  # noqa: E402
from wbgpu import engine, models  # noqa: E402

pytestmark = pytest.mark.gpu


def _r_set(kind, half, rng):
    if kind == 'cube':
        return models.cube_R(half)
    if kind == 'positive':  # no -R partners at all
        return models.cube_R(half)[np.all(models.cube_R(half) >= 0, axis=1)]
    R = models.cube_R(half)  # ragged: a random half of the vectors, shifted off centre
    return R[rng.random(len(R)) < 0.5] + np.array([1, 0, -1])


@pytest.mark.parametrize("prec", [engine.PREC_FP64, engine.PREC_DF64, engine.PREC_DF64C])
@pytest.mark.parametrize("kind,half", [('cube', 1), ('cube', 2), ('cube', 3), ('cube', 5), ('positive', 5),
                                       ('ragged', 2), ('ragged', 4), ('ragged', 6), ('positive', 13)])
def test_transform_against_the_direct_sum(kind, half, prec):
    """sum_R exp(2 pi i R k) X_R per axis: three contractions of at most 27 terms, each rounding within
    27 ulps of the terms' absolute sum (2^-53, 2^-46 in double-float, 2^-24 once for complex64)."""
    rng = np.random.default_rng(half)
    iR = _r_set(kind, half, rng)
    nw, N = 3, (3, 5, 4)
    X = rng.standard_normal((len(iR), nw, nw)) + 1j * rng.standard_normal((len(iR), nw, nw))
    s = wbgpu.System_R.from_arrays(np.eye(3), iR, np.zeros((nw, 3)), {'Ham': X})
    dev = engine.DeviceSystem(s)
    dK = np.array([[0.013, 0.0, 0.07], [0.0, 0.031, 0.002]])
    out, _, nF, keep = engine.r2k(dev, dK, N, set(), True, prec)
    torch.cuda.synchronize()
    raw = out.cpu()
    if prec == engine.PREC_DF64:
        f = torch.view_as_real(raw).contiguous().view(torch.float32).reshape(raw.shape + (4,)).double().numpy()
        got = (f[..., 0] + f[..., 1]) + 1j * (f[..., 2] + f[..., 3])
    else:
        got = raw.numpy().astype(np.complex128)
    j = np.stack(np.meshgrid(*[np.arange(n) for n in N], indexing='ij'), -1).reshape(-1, 3)
    k = np.concatenate([j / np.array(N) + d for d in dK])
    ref = np.einsum('kr,rmn->kmn', np.exp(2j * np.pi * (k @ iR.T)), X)
    eps = {engine.PREC_FP64: 3 * 27 * 2.0 ** -53, engine.PREC_DF64: 3 * 27 * 2.0 ** -46,
           engine.PREC_DF64C: 2.0 ** -24}[prec]
    assert np.abs(got[:, 0] - ref).max() <= eps * np.abs(X).sum(axis=0).max()


def test_fp64_lower_triangles_only_for_exactly_hermitian_matrices():
    """Bases Hermitian bit for bit give lower-triangle fields; one ulp off in one matrix element, or too few
    k-points, keeps the full matrices.  Both agree to rounding."""
    d = models.random_tb(6, 2, np.eye(3) * 2.0, 1.0, 3, centers='random', keys=('Ham', 'AA'))
    grid = lambda s: wbgpu.Grid(s, NKdiv=2, NKFFT=4)
    ef = np.linspace(-1, 1, 21)
    s = wbgpu.System_R.from_dict(d)
    dev = engine.DeviceSystem(s)
    assert dev.hermitian_bases(0.0) == frozenset({'Ham', 'AA'})
    assert engine.fp64_columns(dev, {'V'}, 63)[0] is None and engine.fp64_columns(dev, {'V'}, 64)[0] is not None
    d['XX_R']['Ham'][3, 1, 2] = np.nextafter(d['XX_R']['Ham'][3, 1, 2].real, 9) + 1j * d['XX_R']['Ham'][3, 1, 2].imag
    s2 = wbgpu.System_R.from_dict(d)
    dev2 = engine.DeviceSystem(s2)
    assert dev2.hermitian_bases(0.0) == frozenset({'AA'}) and dev2.hermitian_bases() == frozenset({'Ham', 'AA'})
    calc = lambda: {'ahc': wbgpu.calculators.AHC(Efermi=ef), 'bcd': wbgpu.calculators.BerryDipole_FermiSea(Efermi=ef)}
    a, b = wbgpu.run(s, grid(s), calc()), wbgpu.run(s2, grid(s2), calc())
    for q in a:
        assert np.abs(a[q].data - b[q].data).max() <= 1e-9 * np.abs(a[q].data).max()
