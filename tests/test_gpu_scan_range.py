"""The cumulative scan of a histogram (wbg_scan_finalize) against exact integers: sums that leave an entry's own range
(|sum| < 2^67) while every entry is in it, both signs, runs of one and of several levels a thread."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import _lib, engine  # noqa: E402


@pytest.mark.parametrize("nEF", [1, 5, 256, 257, 3000])
@pytest.mark.parametrize("top", [2.0 ** 10, 2.0 ** 66.9])
def test_cumulative_sums(nEF, top):
    ncomp = 3
    rng = np.random.default_rng(nEF)
    v = rng.uniform(0, top, (nEF, ncomp))
    v[:, 1] *= -1
    v[:, 2] *= rng.choice([-1.0, 1.0], nEF)
    fixed = [int(x.as_integer_ratio()[0] * 2 ** 60 // x.as_integer_ratio()[1]) for x in v.reshape(-1).tolist()]
    words = np.zeros(2 * nEF * ncomp + 1, dtype=np.uint64)
    words[0:-1:2] = [f & (2 ** 64 - 1) for f in fixed]
    words[1:-1:2] = [f >> 64 & (2 ** 64 - 1) for f in fixed]
    hist = torch.from_numpy(words.view(np.int64)).cuda()
    out = torch.empty((nEF, ncomp), dtype=torch.float64, device='cuda')
    st = _lib.load().wbg_scan_finalize(engine._ptr(hist), nEF, ncomp, ctypes.c_double(1.0), engine._ptr(out),
                                       engine._stream())
    _lib.check(st, "wbg_scan_finalize")
    got = out.cpu().numpy()
    sums = np.zeros(ncomp, dtype=object)
    for i in range(nEF):
        sums += np.array(fixed[i * ncomp:(i + 1) * ncomp], dtype=object)
        for c in range(ncomp):
            exact = float(sums[c]) * 2.0 ** -60
            # three roundings at most (the words' values and their sum)
            assert abs(got[i, c] - exact) <= 2.0 ** -51 * abs(exact) + 2.0 ** -60, (i, c)
