"""The sliced rotation above num_wann 32 under a 0 ns bound on every wait: some wait does give up (the products of a stage
take longer than the first look at their barrier), the launch ends, is flagged, and leaves the next one right.  (Up to
num_wann 32 a stage's products end within the first look.)"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import engine  # noqa: E402


@pytest.mark.parametrize("nw,fp", [(48, 1), (82, 2), (128, 1), (128, 2)])
def test_a_wait_runs_out_and_is_flagged(nw, fp):
    lib, nk, nF = engine._lib.load(), 400, 5
    rng = np.random.default_rng(nw)
    U = np.linalg.qr(rng.standard_normal((4, nw, nw)) + 1j * rng.standard_normal((4, nw, nw)))[0]
    X = rng.standard_normal((4, nF, nw, nw)) + 1j * rng.standard_normal((4, nF, nw, nw))
    conv = lambda a: torch.from_numpy(a if fp == 1 else engine._df64_pairs(a)).contiguous().view(torch.complex128)
    Ut = conv(U).reshape(U.shape).repeat(nk // 4, 1, 1).cuda()
    Xt = conv(X).reshape(X.shape).repeat(nk // 4, 1, 1, 1).cuda()
    run = lambda: engine.rotate(Ut, Xt, nF, list(range(nF)), [1] * nF, nw, nk, fp)[0].clone()
    before = run()
    engine.device_flags()
    flags = 0
    try:
        assert lib.wbg_tc_wait_limit(ctypes.c_ulonglong(0)) == 0
        for _ in range(3):
            run()
        flags = engine.device_flags()
    finally:
        assert lib.wbg_tc_wait_limit(ctypes.c_ulonglong(1_000_000_000)) == 0
    assert flags & 1
    after = run()
    torch.cuda.synchronize()
    assert engine.device_flags() == 0
    assert torch.equal(torch.view_as_real(before), torch.view_as_real(after))
