"""FP64 results are the same bits however the blocks of a run are batched."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from wbgpu import models, system as wsys  # noqa: E402
import wbgpu  # noqa: E402

C = wbgpu.calculators
LAT = np.diag([3.0, 3.5, 4.0])


def _same(s, grid, calculators, batches):
    ref = wbgpu.run(s, grid, calculators(), blocks_per_batch=batches[0])
    for nb in batches[1:]:
        got = wbgpu.run(s, grid, calculators(), blocks_per_batch=nb)
        for q in ref:
            assert np.isfinite(ref[q].data).all() and np.abs(ref[q].data).max() > 0, q
            assert np.array_equal(got[q].data, ref[q].data), (q, nb)


@pytest.mark.parametrize("nw,nEF,nomega", [(4, 1, 5), (9, 5, 61), (12, 3, 130)])
def test_frequency_sums(nw, nEF, nomega):
    """Every kind of FP64 frequency sum (real or complex factors and elements), one block of 64 k-points at a time
    and in larger batches."""
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, LAT, seed=nw, keys=('Ham', 'AA', 'SS')))
    opt = dict(Efermi=np.linspace(-0.5, 0.5, nEF) if nEF > 1 else np.array([0.0]), omega=np.linspace(0.0, 4.0, nomega),
               smr_fixed_width=0.05)
    cal = lambda: {'optical': C.OpticalConductivity(**opt), 'shift': C.ShiftCurrent(sc_eta=0.04, **opt),
                   'injection': C.InjectionCurrent(**opt), 'shc': C.SHC(SHC_type='simple', **opt)}
    _same(s, wbgpu.Grid(s, NKdiv=3, NKFFT=(4, 4, 4)), cal, (1, 5, 27))


@pytest.mark.parametrize("div,fft,batches", [(3, (2, 2, 2), (1, 2, 7, 8, 27)),  # 216 k-points, batches below and above 64
                                             (2, (1, 2, 3), (1, 3, 8)),         # 48 k-points
                                             (2, (4, 4, 4), (1, 3, 8))])        # a last batch of other size
def test_batches_around_the_lower_triangle_line(div, fft, batches):
    """Whether a run's FP64 fields are transformed as lower triangles follows from its grid, not from its batches: sums,
    tetrahedra, tabulated values, a server's requests and captured graphs."""
    s = wsys.System_R.from_dict(models.random_tb(6, 1, LAT, seed=3))
    EF = np.linspace(-1.0, 1.0, 11)
    grid = wbgpu.Grid(s, NKdiv=div, NKFFT=fft)
    cal = lambda: {'ahc': C.AHC(Efermi=EF), 'ohmic': C.Ohmic_FermiSurf(Efermi=EF),
                   'tetra': C.AHC(Efermi=EF, tetra=True)}
    _same(s, grid, cal, batches)
    ref = wbgpu.run(s, grid, cal(), blocks_per_batch=batches[-1])
    srv = wbgpu.Server(precision='fp64', max_active=2, max_kpoints=2 * grid.nk_per_block, cuda_graph=True)
    srv.add_system('s', s)
    tickets = [srv.submit('s', grid, cal()) for _ in range(2)]
    srv.run_until_idle()
    for t in tickets:
        for q in ref:
            assert np.array_equal(t.wait()[q].data, ref[q].data), q


@pytest.mark.parametrize("iters,fft", [(0, (2, 2, 3)),  # values of a batch cut on the host
                                       (0, (9, 9, 6)),  # 4 860 rows a batch: packed on the device
                                       (2, (2, 2, 3))])
def test_tabulated_and_refined_batches(monkeypatch, iters, fft):
    """Energies, gradients and curvatures of two blocks at a time through the page-locked buffers, against all at once;
    adaptive refinement."""
    import importlib
    R = importlib.import_module('wbgpu.run')
    s = wsys.System_R.from_dict(models.random_tb(5, 1, LAT, seed=4))
    grid = wbgpu.Grid(s, NKdiv=3, NKFFT=fft)
    EF = np.linspace(-1.0, 1.0, 11)
    if iters:
        go = lambda: {k: v.data for k, v in wbgpu.run(s, grid, {'ahc': C.AHC(Efermi=EF)}, adpt_num_iter=iters).items()}
    else:
        go = lambda: wbgpu.tabulate(s, grid, ('energy', 'band_gradients', 'berry_curvature'))
    a = go()
    monkeypatch.setattr(R, 'choose_batch', lambda *args, **kw: 2)
    b = go()
    for q in a:
        assert np.isfinite(a[q]).all() and np.array_equal(a[q], b[q]), q


@pytest.mark.parametrize("nw", [5, 23])
def test_odd_numbers_of_k_points_and_bands(nw):
    """FP64 pair records of 9 k-points with an odd number of pairs each (the complex elements start on 16 bytes all the
    same), against 18 k-points at once."""
    s = wsys.System_R.from_dict(models.random_tb(nw, 1, LAT, seed=nw, keys=('Ham', 'AA', 'SS')))
    opt = dict(Efermi=np.linspace(-0.5, 0.5, 5), omega=np.linspace(0.0, 4.0, 7), smr_fixed_width=0.05)
    cal = lambda: {'optical': C.OpticalConductivity(**opt), 'shift': C.ShiftCurrent(sc_eta=0.04, **opt),
                   'injection': C.InjectionCurrent(**opt), 'shc': C.SHC(SHC_type='simple', **opt)}
    _same(s, wbgpu.Grid(s, NKdiv=(1, 1, 2), NKFFT=(3, 3, 1)), cal, (2, 1))
