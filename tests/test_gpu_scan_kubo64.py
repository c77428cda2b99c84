"""The parallel Fermi-level scan and the FP64 Kubo sums at their edges."""
import ctypes
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..'))
import wbgpu  # noqa: E402
from oracle import wb_oracle as O  # noqa: E402
from wbgpu import engine, models  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nEF,ncomp", [(1, 1), (2, 3), (31, 9), (255, 3), (256, 1), (257, 27), (1001, 3), (4097, 2)])
def test_scan_finalize_is_the_exact_prefix_sum(nEF, ncomp):
    """Entries of both signs, small and large: the integer prefix sum of the 2^-60 fixed-point words,
    rounded once to double (2^-53 relative, 2^-54 of the largest part) and scaled once."""
    rng = np.random.default_rng(nEF)
    v = [[int(rng.integers(-2 ** 62, 2 ** 62)) << int(rng.integers(0, 40)) for _ in range(ncomp)] for _ in range(nEF)]
    words = np.zeros(2 * nEF * ncomp + 1, dtype=np.uint64)
    for i in range(nEF):
        for c in range(ncomp):
            u = v[i][c] % 2 ** 128
            words[2 * (i * ncomp + c)] = u & (2 ** 64 - 1)
            words[2 * (i * ncomp + c) + 1] = u >> 64
    out = torch.empty((nEF, ncomp), dtype=torch.float64, device='cuda')

    def scan():
        h = torch.from_numpy(words.view(np.int64)).cuda()
        st = engine._lib.load().wbg_scan_finalize(engine._ptr(h), nEF, ncomp, ctypes.c_double(0.5), engine._ptr(out),
                                                  engine._stream())
        assert st == 0
        return out.cpu().numpy()
    got = scan()
    for c in range(ncomp):
        s = 0
        for i in range(nEF):
            s += v[i][c]
            exact = s / 2 ** 61
            assert abs(got[i, c] - exact) <= 2.0 ** -52 * abs(exact) + 2.0 ** -61
    words[-1] = 1
    assert np.isnan(scan()).all()


@pytest.mark.parametrize("nw,nEF,nom", [(6, 3, 65), (5, 5, 130)])
def test_kubo_fp64_tiles(nw, nEF, nom):
    """Every FP64 frequency sum (real and complex factors and elements) across tile edges of 64
    frequencies and 64 / 128 columns, against the oracle: FP64 sums of at most nk nw^2 terms, 1e-12."""
    d = models.random_tb(nw, 1, np.eye(3) * 2.0, 1.0, 5, centers='random', keys=('Ham', 'AA', 'SS'))
    d['XX_R']['SS'] = models.hermitize(d['iRvec'], d['XX_R']['SS'])
    kw = dict(Efermi=np.linspace(-0.5, 0.5, nEF), omega=np.linspace(0.1, 2.0, nom), smr_fixed_width=0.1)
    mk = lambda M, S: {'opt': M.OpticalConductivity(**kw), 'inj': M.InjectionCurrent(smr_type='Gaussian', **kw),
                       'shift': M.ShiftCurrent(sc_eta=0.04, **kw), 'shc': S(SHC_type='simple', kBT=0.02, **kw)}
    s = wbgpu.System_R.from_dict(d)
    got = wbgpu.run(s, wbgpu.Grid(s, NKdiv=1, NKFFT=(2, 3, 2)), mk(wbgpu.calculators, wbgpu.calculators.dynamic.SHC))
    ref = O.run(O.RSystem(d['real_lattice'], d['iRvec'], d['wannier_centers_cart'], d['XX_R']), (1, 1, 1), (2, 3, 2),
                mk(O, O.SHC))
    for k in ref:
        e, r = got[k].data, ref[k].data
        assert e.shape == r.shape and np.max(np.abs(e - r)) < 1e-12 * np.max(np.abs(r)), k
