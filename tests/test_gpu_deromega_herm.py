"""Berry-curvature dipole traces in double-float: k-points with Hermitian V and W (one kernel) and
without (another), against the FP64 kernel on the same complex64 fields."""
import ctypes
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
from wbgpu import _lib, engine  # noqa: E402
from wbgpu.calculators import fixed_values, fixed_words  # noqa: E402

pytestmark = pytest.mark.gpu
# field layout of a random band-basis batch: V 3, W 9, A 3, O 3, dA 9, dO 9
IV, IW, IA, IO, IDA, IDO, NF = 0, 3, 12, 15, 18, 27, 36


def _fields(nw, nk, seed, degenerate):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((nk, NF, nw, nw)) + 1j * rng.standard_normal((nk, NF, nw, nw))
    X = ((X + X.conj().swapaxes(-1, -2)) / 2).astype(np.complex64)
    for b in range(3):  # W = d_b d_d H is symmetric in its directions
        for d in range(b):
            X[:, IW + 3 * b + d] = X[:, IW + 3 * d + b]
    E = np.sort(rng.uniform(-2, 2, (nk, nw)), axis=1)
    if degenerate and nw > 3:
        E[:, nw // 2] = E[:, nw // 2 - 1]
        E[0, 1] = E[0, 0] + 1e-6
    return E, X


def _hist(E, X, arith, internal, external, nEF=41, words=False):
    nk, nw = E.shape
    sc = _lib.Scan(EFmin=-1.0, EFmax=1.0, dEF=2.0 / (nEF - 1), degen_thresh=1e-4, nEF=nEF, reserved=0)
    Et, Xt = torch.from_numpy(E).cuda(), torch.from_numpy(X).cuda()
    h = torch.zeros(fixed_words(9 * nEF), dtype=torch.int64, device='cuda')
    st = _lib.load().wbg_berry_deromega(engine._ptr(Et), engine._ptr(Xt), NF, IV, IA, IO, IW, IDA, IDO, nw, nk,
                                        ctypes.byref(sc), internal, external, engine._ptr(h), arith, engine._stream())
    assert st == 0
    w = h.cpu().numpy()
    return w if words else fixed_values(w, 9 * nEF)


@pytest.mark.parametrize("internal,external", [(1, 1), (1, 0), (0, 1)])
@pytest.mark.parametrize("nw,nk", [(1, 3), (2, 5), (5, 700), (21, 9), (31, 4), (33, 4), (64, 3), (82, 2), (128, 1)])
def test_double_float_against_fp64(nw, nk, internal, external):
    """Random Hermitian fields, bands below, inside and above the window, degenerate groups.  Both kernels
    work to 2^-47 and the same gaps (down to 1e-4, cubed) amplify it: the Hermitian one is no further
    from FP64 than four times the other, which an imaginary 1e-30 on one diagonal element selects."""
    E, X = _fields(nw, nk, 31 * nw + nk, True)
    other = X.copy()
    other[:, IV, 0, 0] += 1e-30j
    got = _hist(E, X, 2, internal, external)
    ref = _hist(E, X.astype(np.complex128), 1, internal, external)
    slow = _hist(E, other, 2, internal, external)
    assert np.abs(got - ref).max() <= 4 * np.abs(slow - ref).max() + 2.0 ** -44 * np.abs(ref).max()


def _entries(words):
    """The fixed-point entries as Python integers."""
    w = words[:-1].view(np.uint64).reshape(-1, 2)
    return [(int(lo) + (int(hi) << 64)) % 2 ** 128 for lo, hi in w]


def test_hermitian_and_other_kpoints_in_one_batch():
    """Every second k-point loses its Hermiticity (V at one element, W at another): each kernel adds exactly
    its own k-points, so the batch's integer histogram is the sum of the two groups' alone."""
    E, X = _fields(12, 40, 5, False)
    X[1::4, IV + 1, 3, 7] += 0.5
    X[3::4, IW + 4, 11, 0] += 0.25j
    whole, even, odd = (_entries(_hist(np.ascontiguousarray(E[s]), np.ascontiguousarray(X[s]), 2, 1, 1, words=True))
                        for s in (slice(None), slice(0, None, 2), slice(1, None, 2)))
    assert any(even) and any(odd)
    assert whole == [(a + b) % 2 ** 128 for a, b in zip(even, odd)]


@pytest.mark.parametrize("nw,nk", [(5, 60), (21, 9), (33, 4), (82, 2)])
def test_fp64_hermitian_kpoints(nw, nk):
    """The same split in FP64: the two FP64 kernels differ by 2^-53 where the double-float one differs by 2^-47
    through the same gaps -- 2^-6 of its distance, with a factor 8 for the different order of the sums."""
    E, X = _fields(nw, nk, 7 * nw + nk, True)
    other = X.astype(np.complex128)
    other[:, IV, 0, 0] += 1e-30j
    general = _hist(E, other, 1, 1, 1)
    got = _hist(E, X.astype(np.complex128), 1, 1, 1)
    df = _hist(E, other.astype(np.complex64), 2, 1, 1)
    assert np.abs(got - general).max() <= 2.0 ** -3 * np.abs(df - general).max() + 2.0 ** -50 * np.abs(general).max()
