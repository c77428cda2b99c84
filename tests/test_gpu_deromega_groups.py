"""The Hermitian-k Berry-curvature dipole under a selection of bands (wbg_band_values) with degenerate groups: against the
general kernel, which takes the k-point when an element that the sums do not read breaks the symmetry."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import _lib, engine  # noqa: E402

DEROMEGA = 4


def _values(E, X, sel, nw, nk):
    f = _lib.FieldIndex(V=0, A=3, O=6, W=9, dA=18, dO=27, B=-1, C=-1)
    P = torch.full((nk, nw, 9), np.nan, dtype=torch.float64, device='cuda')
    Et, Xt, st = torch.from_numpy(E).cuda(), torch.from_numpy(X).cuda(), torch.from_numpy(sel).cuda()
    s = _lib.load().wbg_band_values(engine._ptr(Et), engine._ptr(Xt), 36, ctypes.byref(f), nw, nk, DEROMEGA, 1, 1,
                                    ctypes.c_double(1e-4), engine._ptr(st), engine._ptr(P), 1, engine._stream())
    _lib.check(s, "wbg_band_values")
    return P.cpu().numpy()


@pytest.mark.parametrize("nw", [5, 8, 21, 64, 128])
@pytest.mark.parametrize("part", ['groups', 'parts of groups', 'groups and a sea'])
def test_against_general_kernel(nw, part):
    nk = 6
    rng = np.random.default_rng(nw)
    E = np.sort(rng.uniform(-2, 2, (nk, nw)), axis=1)
    # groups of two and three, the first and the last bands among them
    for k in range(nk):
        for g0, n in ((0, 2), (nw // 2, 3 if nw > 6 else 2), (nw - 2, 2)):
            if k % 2 == 0 or g0:
                E[k, g0:g0 + n] = E[k, g0]
    E = np.maximum.accumulate(E, axis=1)
    X = rng.standard_normal((nk, 36, nw, nw)) + 1j * rng.standard_normal((nk, 36, nw, nw))
    X[:, :3] += X[:, :3].conj().swapaxes(-1, -2)
    W = X[:, 9:18].reshape(nk, 3, 3, nw, nw)
    W = W + W.swapaxes(1, 2)
    X[:, 9:18] = (W + W.conj().swapaxes(-1, -2)).reshape(nk, 9, nw, nw)
    start = np.c_[np.ones((nk, 1), bool), np.diff(E, axis=1) > 1e-4]
    group = np.cumsum(start, axis=1)
    sel = np.zeros((nk, nw), dtype=np.int8)
    for k in range(nk):
        sel[k] = rng.random(group[k].max() + 1)[group[k]] < 0.6
        if part == 'parts of groups':
            sel[k] &= (rng.random(nw) < 0.6)
            sel[k, [0, nw - 1]] = 1  # of the first and of the last group one band
            sel[k, [1, nw - 2]] = 0
        elif part == 'groups and a sea':
            top = np.where(start[k])[0][min(3, start[k].sum() - 1)]
            sel[k, :top] = 2
    general = X.copy()
    general[:, 9, 0, 0] += 1e-3j  # a diagonal element of W: not read, but not Hermitian
    a, b = _values(E, X, sel, nw, nk), _values(E, general, sel, nw, nk)
    assert np.isfinite(a).all() and np.abs(b).max() > 0
    assert (a[sel == 0] == 0).all()
    # sums over nw^2 terms of order |X|^3 / gap^2, rounded in another order
    scale = np.abs(b).max(axis=(1, 2), keepdims=True)
    assert (np.abs(a - b) <= nw * nw * 2.0 ** -50 * scale).all()
