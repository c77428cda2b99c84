"""k-resolved quantities on the GPU path: ``evaluate_k`` and grid tabulation.

Mirrors evaluate_k.py:33-131 (named quantities of evaluate_k.py:9-16) and the Tabulators of
calculators/tabulate.py:21-52: per k-point and band, the trace of the band's degenerate group
(whole band range, no sea group) divided by the group size, for

* ``energy``                          group-averaged E (eV)
* ``band_gradients``                  Re V_nn = dE/dk (eV Angstrom)
* ``berry_curvature``                 Omega (Angstrom^2), internal + external terms
* ``berry_curvature_internal_terms``  internal terms only
* ``berry_curvature_external_terms``  external terms only

Like the reference, a single k-point is a 1x1x1 FFT block with dK = k; a grid tabulates every
block of the grid.  Stages 1-3 are ``engine.band_data`` (FP64 by default), the per-band traces
one ``wbg_berry_tabulate`` launch per term selection.
"""
import ctypes

import numpy as np
import torch

from . import _lib, engine
from .engine import _ptr, _stream

QUANTITIES = ('energy', 'band_gradients', 'berry_curvature', 'berry_curvature_internal_terms',
              'berry_curvature_external_terms')
_TERMS = {'berry_curvature': (1, 1), 'berry_curvature_internal_terms': (1, 0),
          'berry_curvature_external_terms': (0, 1)}


def _check(quantities):
    for q in quantities:
        if q not in QUANTITIES:
            raise ValueError(f"unknown quantity {q}. known quantities are {QUANTITIES}")


def _band_quantities(system, quantities):
    ext = any(_TERMS.get(q, (0, 0))[1] for q in quantities) and not system.force_internal_terms_only
    return {'V', 'A', 'Od'} if ext else {'V'}


def _tab_batch(dev, system, dKs, NKFFT, quantities, precision, degen_thresh, phases=None, block_start=0,
               run_kpoints=None):
    """Per-k, per-band values of `quantities` for a batch of blocks: dict q -> array."""
    bd = engine.band_data(dev, dKs, NKFFT, _band_quantities(system, quantities), precision, phases=phases,
                          block_start=block_start, run_kpoints=run_kpoints)
    nkt, nw = bd.nk_total, bd.nw
    lib = _lib.load()
    iA, iO = bd.index.get('A', 0), bd.index.get('Od', 0)

    def terms(q):  # (internal, external) of one quantity's Omega trace
        internal, external = _TERMS.get(q, (1, 0))
        return internal, external if 'A' in bd.index else 0  # no AA_R: internal terms only

    tabs = {}
    for key in {terms(q) for q in quantities}:
        tab = torch.empty((nkt, nw, 7), dtype=torch.float64, device=bd.E.device)
        st = lib.wbg_berry_tabulate(_ptr(bd.E), _ptr(bd.Xbar), bd.Xbar.shape[1], bd.index['V'], iA, iO, nw, nkt,
                                    ctypes.c_double(degen_thresh), key[0], key[1], _ptr(tab), int(bd.fp64_fields),
                                    _stream())
        _lib.check(st, "wbg_berry_tabulate")
        tabs[key] = tab
    cols = {'energy': slice(0, 1), 'band_gradients': slice(1, 4)}
    # Values and the solver's flag come back with one wait, in page-locked memory (large batches in pageable
    # memory: what was page-locked stays with the process).  A few k-points: the columns in use in one copy, cut
    # on the host; from 4 096 rows on a quantity's columns are packed on the device first (a kernel and a copy
    # a quantity more, some 10 us, against numpy's strided copies: 4.48 -> 3.97 ms for 10 296 k-points x 13 bands)
    pin = nkt * nw * 7 * 8 <= 64 << 20

    def fetch(t):
        h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pin)
        h.copy_(t.contiguous(), non_blocking=True)
        return h

    parts = {}  # (term selection, first and last column) -> host buffer
    for q in quantities:
        c, key = cols.get(q, slice(4, 7)), terms(q)
        if nkt * nw < 4096:
            use = [cols.get(p, slice(4, 7)) for p in quantities if terms(p) == key]
            c = slice(min(u.start for u in use), max(u.stop for u in use))
        if (key, c.start, c.stop) not in parts:
            parts[(key, c.start, c.stop)] = fetch(tabs[key][:, :, c])
    flag = fetch(bd._flag)
    torch.cuda.current_stream(bd.E.device).synchronize()
    engine.check_flag_word(flag)
    out = {}
    for q in quantities:
        c = cols.get(q, slice(4, 7))
        lo, h = next((a, h) for (key, a, e), h in parts.items() if key == terms(q) and a <= c.start and c.stop <= e)
        t = h.numpy()[:, :, c.start - lo:c.stop - lo]
        out[q] = t[:, :, 0] if q == 'energy' else t
    return out


def evaluate_k(system, k=(0., 0., 0.), quantities=(), iband=None, return_single_as_dict=False,
               precision='fp64', degen_thresh=1e-4, device='cuda'):
    """evaluate_k.py:33-131 for the named quantities: values at one k-point (reduced
    coordinates) for the bands `iband` (all by default).  Returns {quantity: array}, or the
    array alone for a single quantity unless return_single_as_dict."""
    quantities = list(quantities)
    _check(quantities)
    engine.require_cuda()
    dev = engine.DeviceSystem(system, device)
    res = _tab_batch(dev, system, np.array([k], dtype=float), [1, 1, 1], quantities, precision, degen_thresh)
    if iband is None:
        iband = np.arange(system.num_wann)
    iband = list(np.atleast_1d(iband))
    result = {q: res[q][0][iband] for q in quantities}
    if len(result) == 1 and not return_single_as_dict:
        return next(iter(result.values()))
    return result


def tabulate(system, grid, quantities=('energy', 'berry_curvature'), ibands=None, precision='fp64',
             degen_thresh=1e-4, device='cuda', dev_system=None):
    """Tabulators over every k-point of `grid` (calculators/tabulate.py:21-52): returns
    {'kpoints': (nk, 3) reduced coordinates, quantity: (nk, nbands[, 3])}, k-points block by
    block, each block in C order of its FFT grid."""
    quantities = list(quantities)
    _check(quantities)
    engine.require_cuda()
    dev = dev_system or engine.DeviceSystem(system, device)
    shifts = grid.block_shifts()
    nk = grid.nk_per_block
    from .run import choose_batch
    nb = choose_batch(dev.nw, nk, len(shifts), _band_quantities(system, quantities), precision)
    precs = engine.phase_precs(precision)
    phases = {p: dev.grid_phases(shifts, grid.FFT, p) for p in precs}
    parts = {q: [] for q in quantities}
    for i0 in range(0, len(shifts), nb):
        res = _tab_batch(dev, system, shifts[i0:i0 + nb], grid.FFT, quantities, precision, degen_thresh,
                         phases=phases, block_start=i0, run_kpoints=grid.nblocks * nk)
        for q in quantities:
            parts[q].append(res[q] if nb >= len(shifts) else res[q].copy())  # (page-locked buffers go round)
    sel = slice(None) if ibands is None else list(np.atleast_1d(ibands))
    out = {q: np.concatenate(parts[q])[:, sel] for q in quantities}
    N = np.array(grid.FFT)
    j = np.stack(np.meshgrid(*[np.arange(n) for n in N], indexing='ij'), -1).reshape(-1, 3)
    out['kpoints'] = np.concatenate([j / N + dK for dK in shifts])
    return out
