"""Register-tiled FP32 rotation at every tile remainder against FP64 products."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
from wbgpu import engine  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [4, 5, 6, 7, 8, 9, 13, 18, 21, 31, 33, 47, 62, 63])
def test_fp32_every_remainder(nw):
    """Plain, Hermitian-part, diagonal and lower-triangle outputs, an invalid selection in between: each sum of
    2 nw products rounds within 2 nw 2^-24 of the absolute sum, twice, below 8 nw 2^-24 max |X|."""
    rng = np.random.default_rng(nw)
    nk, nF = 7, 4
    X = rng.standard_normal((nk, nF, nw, nw)) + 1j * rng.standard_normal((nk, nF, nw, nw))
    X[:, 3] = X[:, 3] + X[:, 3].conj().swapaxes(-1, -2)
    U = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((nk, nw, nw)) + 1j * rng.standard_normal((nk, nw, nw)))[0])
    Xl = X.copy()
    iu = np.triu_indices(nw, 1)
    Xl[:, 3][:, iu[0], iu[1]] = np.nan
    sel, herm = [0, 1, 7, 2, 3, 3], [0, 1, 0, 2, 5, 4]
    got = engine.rotate(torch.from_numpy(U).to(torch.complex64).cuda(), torch.from_numpy(Xl).to(torch.complex64).cuda(),
                        nF, sel, herm, nw, nk, 0)[0].cpu().numpy()
    Y = U.conj().swapaxes(-1, -2)[:, None] @ X @ U[:, None]
    H = (Y + Y.conj().swapaxes(-1, -2)) / 2
    d, tol = np.arange(nw), 8 * nw * 2.0 ** -24 * np.abs(X).max()
    assert np.abs(got[:, 0] - Y[:, 0]).max() < tol and np.abs(got[:, 1] - H[:, 1]).max() < tol
    assert np.isnan(got[:, 2]).all()
    assert np.abs(got[:, 3][:, d, d].real - H[:, 2][:, d, d].real).max() < tol
    assert np.abs(got[:, 4] - H[:, 3]).max() < tol and np.abs(got[:, 5] - Y[:, 3]).max() < tol
    assert np.array_equal(got[:, 1], got[:, 1].conj().swapaxes(-1, -2))


@pytest.mark.parametrize("nw", [8, 12, 16, 20, 24])
@pytest.mark.parametrize("nk", [1, 37, 3001])
def test_wide_loads_keep_the_bits(nw, nk):
    """num_wann a multiple of four: the kernel of 16-byte pieces against the general one, which operands off a
    16-byte boundary take (a strided U of odd distance the same way), every input and output mode."""
    import ctypes
    lib, nF = engine._lib.load(), 6
    g = torch.Generator(device='cuda')
    g.manual_seed(nw)
    X = torch.view_as_complex(torch.randn(nk, nF, nw, nw, 2, device='cuda', generator=g))
    X[:, 3:5][..., torch.ones(nw, nw, dtype=torch.bool, device='cuda').triu(1)] = float('nan')  # never read
    U = torch.view_as_complex(torch.randn(nk, nw, nw, 2, device='cuda', generator=g))
    sel = torch.tensor([0, 1, 2, 3, 4, 77], dtype=torch.int32, device='cuda')  # the last: no such field
    herm = torch.tensor([0, 1, 2, 5, 6, 0], dtype=torch.int32, device='cuda')

    def run(shift, gap):
        x = torch.zeros(X.numel() + 2, dtype=torch.complex64, device='cuda')
        x[shift:shift + X.numel()] = X.reshape(-1)
        u = torch.zeros(nk, nw * nw + gap, dtype=torch.complex64, device='cuda')
        u[:, :nw * nw] = U.reshape(nk, -1)
        out = torch.zeros((nk, nF, nw, nw), dtype=torch.complex64, device='cuda')
        st = lib.wbg_rotate(engine._ptr(u), nw * nw + gap, ctypes.c_void_p(x.data_ptr() + 8 * shift), nF,
                            engine._ptr(sel), engine._ptr(herm), nF, engine._ptr(out), nw, nk, 0, engine._stream())
        assert st == 0
        return torch.view_as_real(out).cpu().numpy()
    wide = run(0, 0)
    assert np.isfinite(wide[:, :5]).all() and np.isnan(wide[:, 5]).all()
    for other in (run(1, 0), run(0, 1), run(0, 2)):
        assert np.array_equal(wide, other, equal_nan=True)
