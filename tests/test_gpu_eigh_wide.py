"""Eigensolver for n > 32 (a block per matrix) and small batches (a warp per matrix in the QL sweep):
residuals and orthogonality, and the same matrix in batches that take the different launches."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
from wbgpu import engine  # noqa: E402

pytestmark = pytest.mark.gpu
PRECISE_DF = 3 | engine.EIGH_PRECISE_VECTORS | engine.EIGH_DF64_VECTORS


def _solve(H, mode):
    nk, n = H.shape[:2]
    T = torch.from_numpy(engine._df64_pairs(H)).contiguous().view(torch.complex128).reshape(H.shape) if mode & 3 == 3 \
        else torch.from_numpy(H)
    U = torch.empty((nk, n, n), dtype=torch.complex128, device='cuda')
    E, U, f = engine.eigh(T.cuda(), n * n, n, nk, mode=mode, U=U)
    assert int(f.item()) == 0
    if mode & 3 == 3:
        w = torch.view_as_real(U.cpu()).contiguous().view(torch.float32).reshape(nk, n, n, 4).double().numpy()
        return E.cpu().numpy(), (w[..., 0] + w[..., 1]) + 1j * (w[..., 2] + w[..., 3])
    return E.cpu().numpy(), U.cpu().numpy()


@pytest.mark.parametrize("mode", [1, PRECISE_DF])
@pytest.mark.parametrize("n", [2, 31, 33, 47, 64, 65, 96, 127, 128])
def test_residual_and_batches(n, mode):
    """|H u - E u| and |U^H U - 1| within 100 n eps |H| (eps 2^-53 / 2^-46; random matrices, whose smallest gap
    of n = 128 is above 1e-4 |H| / n), and bit-identical pairs for a matrix in a batch of 5 and of 700."""
    rng = np.random.default_rng(n)
    H = rng.standard_normal((5, n, n)) + 1j * rng.standard_normal((5, n, n))
    H = H + H.conj().swapaxes(1, 2)
    H[4] = np.diag(np.arange(n) % 7 - 3.0)  # diagonal, degenerate
    E, U = _solve(H, mode)
    eps = 2.0 ** -53 if mode == 1 else 2.0 ** -46
    norm = np.abs(np.linalg.eigvalsh(H)).max()
    assert np.abs(H @ U - U * E[:, None, :]).max() < 100 * n * eps * norm
    assert np.abs(E - np.linalg.eigvalsh(H)).max() < 100 * n * eps * norm
    g = np.abs(U[:4].conj().swapaxes(1, 2) @ U[:4] - np.eye(n)).max()
    gap = np.diff(E[:4], axis=1).min() if n > 1 else norm
    assert g < 100 * n * eps * max(1.0, norm / gap)
    big = np.repeat(H, 140, axis=0)
    Eb, Ub = _solve(big, mode)
    assert np.array_equal(Eb.reshape(5, 140, n)[:, 77], E) and np.array_equal(Ub.reshape(5, 140, n, n)[:, 77], U)
