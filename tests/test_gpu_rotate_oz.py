"""FP64 and double-float rotation on the fp16 tensor cores (8-bit slices): against extended-precision
products at the edges of its tiles, and the values it has to pass on."""
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
from wbgpu import engine  # noqa: E402

pytestmark = pytest.mark.gpu
MODES = [0, 1, 2, 5, 4]


def _case(nw, nk, nF, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((nk, nF, nw, nw)) + 1j * rng.standard_normal((nk, nF, nw, nw))
    X[:, 1] *= 1e-200
    X[:, 2] *= 1e150
    X[:, 3:5] = X[:, 3:5] + X[:, 3:5].conj().swapaxes(-1, -2)
    U = np.linalg.qr(rng.standard_normal((nk, nw, nw)) + 1j * rng.standard_normal((nk, nw, nw)))[0]
    return np.ascontiguousarray(U), X


def _exact(U, X):
    Ul, Xl = U.astype(np.clongdouble)[:, None], X.astype(np.clongdouble)
    t = np.einsum('kfij,kfjn->kfin', Xl, np.broadcast_to(Ul, Xl.shape))
    return np.einsum('kfim,kfin->kfmn', np.broadcast_to(Ul.conj(), Xl.shape), t)


def _worst(got, Y):
    """Largest error per field over its largest element, in each output mode's elements."""
    nw = Y.shape[-1]
    H = (Y + Y.conj().swapaxes(-1, -2)) / 2
    d, out = np.arange(nw), []
    for f, m in enumerate(MODES):
        r = Y[:, f] if m & 3 == 0 else H[:, f]
        e = np.abs((got[:, f][:, d, d].real - r[:, d, d].real) if m & 3 == 2 else got[:, f] - r)
        out.append(float(np.max(e) / np.max(np.abs(Y[:, f]))))
    return max(out)


@pytest.mark.parametrize("nw", [4, 5, 8, 9, 16, 17, 24, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128])
def test_fp64_against_extended_precision(nw):
    """Operands enter with >= 54 bits of their matrix's largest element and each GEMM rounds once: an
    element is off by at most sqrt(2 nw) 2^-54 (operands) per GEMM and 2^-53 (output) of the largest one,
    times the ratio 2 of a power of two to the largest element: 2^-53 (1 + 2 sqrt(2 nw)) bounds it, and
    stays below the n eps of an FP64 dot product."""
    U, X = _case(nw, 3, 5, nw)
    Xl = X.copy()
    iu = np.triu_indices(nw, 1)
    Xl[:, 3:5][..., iu[0], iu[1]] = np.nan
    got, _ = engine.rotate(torch.from_numpy(U).cuda(), torch.from_numpy(Xl).cuda(), 5, [0, 1, 2, 3, 4], MODES, nw, 3,
                           1)
    assert _worst(got.cpu().numpy(), _exact(U, X)) < 2.0 ** -53 * (1 + 2 * np.sqrt(2 * nw))


@pytest.mark.parametrize("nw", [33, 64, 82, 128])
def test_double_float_is_complex64_rounding(nw):
    U, X = _case(nw, 2, 5, nw)
    X[:, 1] *= 1e190
    X[:, 2] *= 1e-145
    df = lambda a: torch.from_numpy(engine._df64_pairs(a)).contiguous().view(torch.complex128).reshape(a.shape).cuda()
    got, _ = engine.rotate(df(U), df(X), 5, [0, 1, 2, 3, 4], MODES, nw, 2, 2)
    assert got.dtype == torch.complex64
    # one rounding to 24 bits of each part, and the double-float operands' 2^-47 under it
    assert _worst(got.cpu().numpy().astype(np.complex128), _exact(U, X)) < 2.0 ** -24


@pytest.mark.parametrize("nw", [4, 13, 32, 48])
def test_special_values(nw):
    """Zero fields stay zero, a non-finite element makes its field NaN and leaves the others alone, a
    selection outside the input is NaN, a non-finite U makes its k-point NaN."""
    U, X = _case(nw, 4, 5, 7 * nw)
    X[0, 0] = 0
    X[1, 0, nw - 1, 0] = np.inf
    X[2, 4, 0, nw - 1] = np.nan
    U2 = U.copy()
    U2[3, nw - 1, nw - 1] = np.nan
    sel = [0, 3, 9, 4, 0]
    herm = [0, 1, 0, 0, 1]
    got = engine.rotate(torch.from_numpy(U2).cuda(), torch.from_numpy(X).cuda(), 5, sel, herm, nw, 4, 1)[0].cpu().numpy()
    bad = np.isnan(got).all(axis=(2, 3))
    fin = np.isfinite(got).all(axis=(2, 3))
    expect = np.zeros((4, 5), dtype=bool)
    expect[:, 2] = expect[3] = True
    expect[1, 0] = expect[1, 4] = expect[2, 3] = True
    assert np.array_equal(bad, expect) and np.array_equal(fin, ~expect)
    assert (got[0, 0] == 0).all() and (got[0, 4] == 0).all()


def test_many_fields_and_strided_u():
    """More fields than one launch keeps, U matrices with a gap between them."""
    nw, nk, nF = 4, 2, 300
    rng = np.random.default_rng(3)
    X = rng.standard_normal((nk, nF, nw, nw)) + 1j * rng.standard_normal((nk, nF, nw, nw))
    Up = rng.standard_normal((nk, nw + 1, nw)) + 1j * rng.standard_normal((nk, nw + 1, nw))
    lib = engine._lib.load()
    Ut, Xt = torch.from_numpy(Up).cuda(), torch.from_numpy(X).cuda()
    sel = torch.arange(nF, dtype=torch.int32).cuda()
    herm = torch.zeros(nF, dtype=torch.int32).cuda()
    out = torch.empty((nk, nF, nw, nw), dtype=torch.complex128, device='cuda')
    st = lib.wbg_rotate(engine._ptr(Ut), (nw + 1) * nw, engine._ptr(Xt), nF, engine._ptr(sel), engine._ptr(herm), nF,
                        engine._ptr(out), nw, nk, 1, engine._stream())
    assert st == 0
    Y = _exact(np.ascontiguousarray(Up[:, :nw]), X)
    assert float(np.abs(out.cpu().numpy() - Y).max() / np.abs(Y).max()) < 2.0 ** -53 * (1 + 2 * np.sqrt(2 * nw))


@pytest.mark.parametrize("nw,fp", [(32, 1), (48, 1), (82, 2)])
def test_waits_that_run_out(nw, fp):
    """With a 0 ns bound on every wait the blocks that find a barrier incomplete give up together, drain their
    products and return; with the normal bound the same call then gives the same bits as before."""
    import ctypes
    lib, nk = engine._lib.load(), 400
    U, X = _case(nw, 4, 5, nw)
    X[:, 1:3] = X[:, 3:5]  # double-float holds the range of floats
    conv = lambda a: torch.from_numpy(a if fp == 1 else engine._df64_pairs(a)).contiguous().view(torch.complex128)
    Ut = conv(U).reshape(U.shape).repeat(nk // 4, 1, 1).cuda()
    Xt = conv(X).reshape(X.shape).repeat(nk // 4, 1, 1, 1).cuda()
    run = lambda: engine.rotate(Ut, Xt, 5, [0, 1, 2, 3, 4], MODES, nw, nk, fp)[0].clone()
    diag = lambda a: torch.view_as_real(a.diagonal(dim1=-2, dim2=-1).contiguous())
    before = run()
    engine.device_flags()
    try:
        assert lib.wbg_tc_wait_limit(ctypes.c_ulonglong(0)) == 0
        run()
        torch.cuda.synchronize()
        engine.device_flags()  # whether a block gave up depends on timing
    finally:
        assert lib.wbg_tc_wait_limit(ctypes.c_ulonglong(1_000_000_000)) == 0
    after = run()
    torch.cuda.synchronize()
    assert engine.device_flags() == 0
    assert torch.equal(torch.view_as_real(before[:, [0, 1, 3]]), torch.view_as_real(after[:, [0, 1, 3]]))
    assert torch.equal(diag(before), diag(after))
