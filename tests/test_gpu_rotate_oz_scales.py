"""The sliced rotation's accuracy where U mixes only some of the bands: blocks of very different size in one field keep
the accuracy that they have alone, component by component."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
from wbgpu import engine  # noqa: E402

pytestmark = pytest.mark.gpu
HERM = [0, 1, 5, 2]


def _blocks(nw, nk, scales, seed):
    """U unitary inside the blocks, its columns in mixed order (as eigenvectors sorted by energy), X block-diagonal,
    the blocks' rows interleaved; the block of each row of X and U and of each column of U."""
    rng = np.random.default_rng(seed)
    row = np.arange(nw) % len(scales)
    col = rng.permutation(row)
    U = np.zeros((nk, nw, nw), dtype=complex)
    X = np.zeros((nk, len(HERM), nw, nw), dtype=complex)
    for b, sc in enumerate(scales):
        i, j = np.where(row == b)[0], np.where(col == b)[0]
        n = len(i)
        q = np.linalg.qr(rng.standard_normal((nk, n, n)) + 1j * rng.standard_normal((nk, n, n)))[0]
        x = sc * (rng.standard_normal((nk, len(HERM), n, n)) + 1j * rng.standard_normal((nk, len(HERM), n, n)))
        x[:, 2:] = x[:, 2:] + x[:, 2:].conj().swapaxes(-1, -2)
        U[:, i[:, None], j[None, :]] = q
        X[:, :, i[:, None], i[None, :]] = x
    return U, X, col


def _check(nw, nk, scales, fp, tol, seed):
    U, X, col = _blocks(nw, nk, scales, seed)
    if fp == 2:  # what the double-float operands hold
        h = lambda a: a.astype(np.float32).astype(np.float64)
        part = lambda a: h(a) + h(a - h(a))
        U, X = (part(a.real) + 1j * part(a.imag) for a in (U, X))
    Xin = X.copy()
    iu = np.triu_indices(nw, 1)
    Xin[:, 2][..., iu[0], iu[1]] = np.nan  # a lower triangle
    conv = lambda a: torch.from_numpy(a if fp == 1 else engine._df64_pairs(a)).contiguous().view(torch.complex128)
    got = engine.rotate(conv(U).reshape(U.shape).cuda(), conv(Xin).reshape(X.shape).cuda(), 4, [0, 1, 2, 3], HERM, nw, nk,
                        fp)[0].cpu().numpy().astype(np.clongdouble)
    Ul, Xl = U.astype(np.clongdouble)[:, None], X.astype(np.clongdouble)
    Y = np.einsum('kfim,kfin->kfmn', np.broadcast_to(Ul.conj(), X.shape),
                  np.einsum('kfij,kfjn->kfin', Xl, np.broadcast_to(Ul, X.shape)))
    H = (Y + Y.conj().swapaxes(-1, -2)) / 2
    d = np.arange(nw)
    for f, m in enumerate(HERM):
        r, g = (Y if m & 3 == 0 else H)[:, f], got[:, f]
        for b in range(len(scales)):
            j = np.where(col == b)[0]
            big = np.abs(r[:, j[:, None], j[None, :]]).max()
            if m & 3 == 2:  # the diagonal
                assert np.abs(g[:, j, j] - r[:, j, j]).max() <= tol * big, (nw, f, b)
                continue
            err = np.abs(g - r)[:, j[:, None], j[None, :]].max()
            assert err <= tol * big, (nw, f, b, float(err / big))
        if m & 3 != 2:
            assert (g[:, col[:, None] != col[None, :]] == 0).all(), (nw, f)


@pytest.mark.parametrize("nw", [4, 7, 8, 13, 16, 21, 24, 31, 32, 33, 48, 64, 82, 96, 127, 128])
def test_fp64_blocks(nw):
    """The bound of a dense field (test_gpu_rotate_oz.py) for each block by itself: 2^-53 (1 + 2 sqrt(2 nw)) of the
    block's largest element, for blocks 1, 1e-8, 1e120 and 1e-150."""
    _check(nw, 3, [1.0, 1e-8] if nw < 8 else [1.0, 1e-8, 1e120, 1e-150], 1, 2.0 ** -53 * (1 + 2 * np.sqrt(2 * nw)), nw)


@pytest.mark.parametrize("nw", [33, 64, 82, 128])
def test_double_float_blocks(nw):
    """Each block within one rounding to complex64 (blocks 1, 1e-7, 1e15 and 1e-20)."""
    _check(nw, 2, [1.0, 1e-7, 1e15, 1e-20], 2, 2.0 ** -24, nw)
