"""Tetrahedron accumulation with lanes on Fermi levels: level counts around the 8 lanes of a band, one band
and more than 32, windows that start and end inside and outside the levels."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))
sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..'))
import wbgpu  # noqa: E402
from oracle import wb_oracle as O  # noqa: E402
from wbgpu import models  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ['fp64', 'mixed'])
@pytest.mark.parametrize("nw,nEF,top", [(1, 2, 0.5), (3, 7, 0.2), (3, 8, 3.0), (4, 9, 1.0), (33, 16, 1.0), (3, 300, 2.0)])
def test_level_counts(nw, nEF, top, precision):
    """CumDOS, Ohmic (der 1) and AHC against the oracle: FP64 to 1e-9 (the derivative divides by gaps down to
    1e-3 of the bands' width), the mixed path's FP32 weights and fields to 2e-5 of the largest level."""
    d = models.random_tb(nw, 1, np.eye(3) * 1.5, 1.0, 40 + nw, centers='random', keys=('Ham', 'AA'))
    ef = np.linspace(-top, top, nEF)
    mk = lambda M: {'cumdos': M.CumDOS(Efermi=ef, tetra=True), 'ohmic': M.Ohmic_FermiSurf(Efermi=ef, tetra=True),
                    'ahc': M.AHC(Efermi=ef, tetra=True)}
    s = wbgpu.System_R.from_dict(d)
    got = wbgpu.run(s, wbgpu.Grid(s, NKdiv=(1, 2, 1), NKFFT=(3, 2, 3)), mk(wbgpu.calculators), precision=precision)
    ref = O.run(O.RSystem(d['real_lattice'], d['iRvec'], d['wannier_centers_cart'], d['XX_R']), (1, 2, 1), (3, 2, 3),
                mk(O))
    tol = 1e-9 if precision == 'fp64' else 2e-5
    for k in ref:
        e, r = got[k].data, ref[k].data
        assert np.abs(e - r).max() <= tol * max(np.abs(r).max(), 1e-12), k
