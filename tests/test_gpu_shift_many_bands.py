"""The shift current of more bands than its table of principal-value factors holds (num_wann 167 in FP64, 238 in FP32):
bands without matrix elements, far above, change nothing."""
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import engine  # noqa: E402
from wbgpu.calculators import ShiftCurrent  # noqa: E402


@pytest.mark.parametrize("nw,fp64", [(128, True), (166, True), (170, True), (200, False), (240, False)])
def test_padded_with_empty_bands(nw, fp64):
    n, nk, nF = 9, 2, 24
    rng = np.random.default_rng(nw)
    E = np.sort(rng.uniform(-1, 1, (nk, n)), axis=1)
    X = rng.standard_normal((nk, nF, n, n)) + 1j * rng.standard_normal((nk, nF, n, n))
    X = X + X.conj().swapaxes(-1, -2)
    system = types.SimpleNamespace(force_internal_terms_only=False)

    def run(E, X):
        m = E.shape[1]
        Xt = torch.from_numpy(X if fp64 else X.astype(np.complex64)).cuda()
        bd = engine.BandData(torch.from_numpy(E).cuda(), None, Xt, {'V': 0, 'A': 3, 'W': 6, 'dA': 15}, 1, nk, m, fp64)
        c = ShiftCurrent(Efermi=np.array([-0.2, 0.3]), omega=np.linspace(0.1, 2.0, 7), smr_fixed_width=0.1, sc_eta=0.05)
        c.reset('cuda')
        c.accumulate(bd, system)
        return c.result(1.0, nk).data

    ref = run(E, X)
    Ep = np.concatenate([E, 1e3 + np.tile(np.arange(nw - n, dtype=float), (nk, 1))], axis=1)
    Xp = np.zeros((nk, nF, nw, nw), dtype=complex)
    Xp[:, :, :n, :n] = X
    got = run(np.ascontiguousarray(Ep), Xp)
    assert np.abs(ref).max() > 0
    # the same terms in the same order; FP64 divisions and sums may round differently once each, FP32 ones too
    assert np.abs(got - ref).max() < (1e-13 if fp64 else 1e-5) * np.abs(ref).max()
