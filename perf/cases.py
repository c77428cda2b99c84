"""What the performance of this framework is measured on: calls of its public entry points.

A case names what a user asks for (`kind`), the model (`nw` Wannier functions, R-vectors in
[-half, half]^3, lattice), the k-points (`div` blocks of `fft` points per axis, of which the
first `blocks` are run, 0: all), the energy axes and the arithmetic (`precision` of run()).
A program that integrates over a grid has in hand: the System_R, its DeviceSystem (the matrices
resident on the GPU), the Grid and the calculators; one pass is one run() / tabulate() /
evaluate_k() call, which returns host arrays, as for every user.

Models are the random tight-binding models of the benchmark and the tests (wbgpu.models):
X_R ~ CN(0, 1) exp(-|R| / decay).  The benchmark's num_wann = 32 system has 1 233 R-vectors after
its Wigner-Seitz replica search, a set-up step on the host; [-5, 5]^3 (1 331) stands for it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), '..', 'wannier-berri_gb300'))

import wbgpu  # noqa: E402
from wbgpu import models  # noqa: E402
from wbgpu.calculators import (AHC, BerryDipole_FermiSea, BerryDipole_FermiSurf, DOS, JDOS, Morb, Ohmic_FermiSurf,  # noqa: E402
                               OpticalConductivity, ShiftCurrent)

TAB = ('energy', 'band_gradients', 'berry_curvature')


def case(name, kind, nw, half, div, fft, blocks=0, nef=0, nomega=0, precision='fp64', tetra=False, lattice='triclinic',
         soc=False):
    d = dict(kind=kind, nw=nw, half=half, div=div, fft0=fft[0], fft1=fft[1], fft2=fft[2], blocks=blocks, nef=nef,
             nomega=nomega, precision=precision, tetra=tetra, lattice=lattice, soc=soc)
    return dict(name=name, **d) if name else d


def listed():
    return [
        # one k-point of a band path: interactive use, the smallest call there is
        case('bands nw8', 'bands', 8, 2, 1, (1, 1, 1), lattice='cubic'),
        # a quick look at a small model in the default precision: latency and launches
        case('ahc nw8 8x4^3 fp64', 'ahc', 8, 2, 2, (4, 4, 4), nef=101, lattice='cubic'),
        # the small-model benchmark configuration: anomalous Hall conductivity on a 48^3 grid
        case('ahc nw8 48^3 mixed', 'ahc', 8, 2, 6, (8, 8, 8), nef=501, precision='mixed', lattice='cubic'),
        # the headline workload: four 24^3 blocks of the 192^3 grid, 1 001 Fermi levels
        case('ahc nw32 4x24^3 mixed', 'ahc', 32, 5, 8, (24, 24, 24), blocks=4, nef=1001, precision='mixed'),
        # the same in the default precision (one block)
        case('ahc nw32 24^3 fp64', 'ahc', 32, 5, 8, (24, 24, 24), blocks=1, nef=1001),
        # tetrahedron integration: corner energies besides the eigenvectors
        case('tetra nw32 24^3 mixed', 'ahc', 32, 4, 2, (12, 12, 12), nef=1001, precision='mixed', tetra=True),
        # a mid-size material in the default precision on an anisotropic grid: transport and moments
        case('transport nw18 fp64', 'transport', 18, 3, 2, (9, 7, 10), nef=201),
        # k-resolved tabulation (Fermi surfaces, curvature maps), odd sizes
        case('tabulate nw13 fp64', 'tabulate', 13, 2, 2, (11, 9, 13)),
        # nonlinear optics in the default precision
        case('shift current nw12 fp64', 'photo', 12, 2, 2, (5, 6, 7), nef=3, nomega=61),
        # a system of the multi-system benchmark: AHC and Berry-curvature dipole, 16^3
        case('dipole nw21 16^3 mixed', 'dipole', 21, 2, 1, (16, 16, 16), nef=201, precision='mixed'),
        # one of its large systems
        case('dipole nw82 8^3 mixed', 'dipole', 82, 2, 1, (8, 8, 8), nef=201, precision='mixed'),
        # the spin-orbit benchmark configuration: optical conductivity at 11 x 400 and AHC, one 8^3 block
        case('optical nw96 8^3 mixed', 'optical', 96, 3, 12, (8, 8, 8), blocks=1, nef=11, nomega=400,
             precision='mixed', soc=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(['ahc', 'ahc', 'ahc', 'transport', 'tabulate', 'dipole', 'optical', 'photo', 'bands'])
    # num_wann and the k-points of the range each kind covers; nk nw^3 stays below the largest listed case's
    lo, hi, nmax, total = {'ahc': (4, 128, 110592, 55296 * 32 ** 3), 'transport': (4, 64, 20000, 5040 * 18 ** 3),
                           'tabulate': (4, 64, 20000, 10296 * 24 ** 3), 'dipole': (4, 128, 8000, 512 * 82 ** 3),
                           'optical': (8, 128, 8000, 512 * 96 ** 3), 'photo': (4, 24, 3000, 1680 * 12 ** 3),
                           'bands': (4, 128, 1, 128 ** 3)}[kind]
    nw = int(round(_log(rng, lo, hi)))
    half = rng.randint(1, 5 if nw <= 40 else 3 if nw <= 100 else 2)
    if kind == 'bands':
        return case(None, kind, nw, half, 1, (1, 1, 1), lattice=rng.choice(['cubic', 'triclinic']))
    nk = max(8.0, _log(rng, 64, max(65, min(nmax, total / nw ** 3))))
    div = rng.choice([1, 2, 3]) if nk >= 216 else 1
    edge = (nk / div ** 3) ** (1 / 3)
    fft = tuple(max(1, min(24, int(edge * rng.uniform(0.8, 1.15)))) for _ in range(3))
    nef, nomega = rng.choice([51, 101, 201, 501, 1001]), 0
    if kind == 'optical':
        nef, nomega = rng.randint(1, 11), rng.randint(20, 400)
    elif kind == 'photo':
        nef, nomega = rng.randint(1, 5), rng.randint(10, 61)
    elif kind == 'tabulate':
        nef = 0
    return case(None, kind, nw, half, div, fft, nef=nef, nomega=nomega,
                precision=rng.choice(['fp64', 'mixed']) if kind not in ('tabulate', 'photo') else 'fp64',
                tetra=kind == 'ahc' and rng.random() < 0.25, lattice=rng.choice(['cubic', 'triclinic']),
                soc=kind == 'optical' and nw % 2 == 0)


# ---------------------------------------------------------------------------------------
def _model(c, seed):
    """The case's model as plain arrays (real_lattice, iRvec, wannier_centers_cart, XX_R)."""
    rng = np.random.default_rng(seed + 7)
    cubic = c['lattice'] == 'cubic'
    lat = np.eye(3) if cubic else models.triclinic_lattice(rng)
    keys = ('Ham', 'AA', 'BB', 'CC') if c['kind'] == 'transport' else ('Ham', 'AA')
    return models.random_tb(c['nw'], c['half'], lat, 1.0 if cubic or c['soc'] else 1.5, seed,
                            centers='zero' if cubic else 'random', keys=keys, soc_pairs=c['soc'])


def _axes(c):
    top = 1.0 if c['kind'] in ('dipole', 'optical', 'photo') else 2.0
    return np.linspace(-top, top, c['nef']) if c['nef'] > 1 else np.array([0.0]), np.linspace(0.0, 4.0, max(c['nomega'], 1))


def _kgrid(c):
    """Block shifts that the case runs, (n, 3), and the block's FFT grid."""
    fft = np.array([c['fft0'], c['fft1'], c['fft2']])
    g = np.stack(np.meshgrid(*[np.arange(c['div'])] * 3, indexing='ij'), axis=-1).reshape(-1, 3)
    if c['blocks']:
        g = g[:c['blocks']]
    return g / c['div'] / fft[None, :], fft


def prepare(c, seed):
    system = wbgpu.System_R.from_dict(_model(c, seed))
    if c['kind'] == 'bands':
        return dict(kind='bands', system=system, k=np.random.default_rng(seed).uniform(0, 1, 3))
    fft = (c['fft0'], c['fft1'], c['fft2'])
    s = dict(kind=c['kind'], system=system, grid=wbgpu.Grid(system, NKdiv=c['div'], NKFFT=fft),
             dev=wbgpu.engine.DeviceSystem(system), precision=c['precision'],
             blocks=list(range(c['blocks'])) if c['blocks'] else None)
    ef, om = _axes(c)
    opt = dict(Efermi=ef, omega=om, smr_fixed_width=0.05)
    s['calculators'] = {
        'ahc': lambda: {'ahc': AHC(Efermi=ef, tetra=c['tetra'])},
        'transport': lambda: {'dos': DOS(Efermi=ef), 'ohmic': Ohmic_FermiSurf(Efermi=ef), 'morb': Morb(Efermi=ef),
                              'dipole': BerryDipole_FermiSurf(Efermi=ef)},
        'dipole': lambda: {'ahc': AHC(Efermi=ef), 'dipole': BerryDipole_FermiSea(Efermi=ef)},
        'optical': lambda: {'ahc': AHC(Efermi=ef), 'optical': OpticalConductivity(**opt)},
        'photo': lambda: {'jdos': JDOS(**opt), 'shift': ShiftCurrent(sc_eta=0.04, **opt)},
        'tabulate': lambda: None,
    }[c['kind']]()
    return s


def run(s):
    if s['kind'] == 'bands':
        return wbgpu.evaluate_k(s['system'], k=s['k'], quantities=TAB)
    if s['kind'] == 'tabulate':
        r = wbgpu.tabulate(s['system'], s['grid'], TAB, precision=s['precision'], dev_system=s['dev'])
        return {q: r[q] for q in TAB}
    r = wbgpu.run(s['system'], s['grid'], s['calculators'], precision=s['precision'], dev_system=s['dev'],
                  blocks=s['blocks'])
    return {k: v.data for k, v in r.items()}


# nw x nw fields of each kind that go to the band basis
_FIELDS = {'bands': 9, 'tabulate': 9, 'ahc': 9, 'transport': 15, 'dipole': 36, 'optical': 9, 'photo': 24}


def work(c):
    """Matrices read once and results written once; eigenproblems at 24 nw^3, U^dagger X U at 16 nw^3
    a field and the last axis of the R -> k transform at 8 (2 half + 1) a matrix element."""
    nw, nR = c['nw'], (2 * c['half'] + 1) ** 3
    nk = int(np.prod([c['fft0'], c['fft1'], c['fft2']])) * (c['blocks'] or c['div'] ** 3)
    nF = _FIELDS[c['kind']]
    nbase = {'transport': 10}.get(c['kind'], 4)
    out = {'bands': 7 * nw, 'tabulate': 7 * nw * nk, 'ahc': 3 * c['nef'], 'transport': 22 * c['nef'],
           'dipole': 12 * c['nef'], 'optical': c['nef'] * (3 + 18 * c['nomega']),
           'photo': 28 * c['nef'] * c['nomega']}[c['kind']]
    flops = nk * (24.0 * nw ** 3 + 16.0 * nF * nw ** 3 + 8.0 * (2 * c['half'] + 1) * (1 + nF) * nw * nw)
    if c['tetra']:
        flops += nk * (16.0 / 3.0 * nw ** 3 + 8.0 * (2 * c['half'] + 1) * nw * nw)
    if c['nomega']:  # pairs across the Fermi level, each at every frequency
        flops += nk * nw * nw / 2 * c['nomega'] * (36.0 if c['kind'] == 'optical' else 60.0)
    return {'bytes': 16.0 * nbase * nR * nw * nw + 8.0 * out, 'flops': flops}


# ---------------------------------------------------------------------------------------
# The same quantities in plain 64-bit torch: direct sums over R, torch.linalg.eigh, the formulas
# of single (non-degenerate) bands -- the models have no degeneracies.
# ---------------------------------------------------------------------------------------
_E, _HBAR, _ANG = 1.602176634e-19, 6.62607015e-34 / (2 * math.pi), 1e-10
_AHC = -_E ** 2 / _HBAR / _ANG
_OHMIC = _E ** 2 / _HBAR / _ANG * 1e-15 * _E / _HBAR
_SHIFT = _HBAR / _E * math.pi * _E ** 3 / (4 * _HBAR ** 2)
_BOHR, _HARTREE = 0.529177210544, 27.211386245981
_ALPHA, _BETA = [1, 2, 0], [2, 0, 1]


class _Bands:
    """Band-basis matrices at a list of k-points: [k, m, n, ...] complex128."""

    def __init__(self, d, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(dev)
        self.R = t(d['iRvec'].astype(float))
        self.nw = d['XX_R']['Ham'].shape[1]
        w = d['wannier_centers_cart']
        cR = d['iRvec'].dot(d['real_lattice'])
        self.w = t(cR[:, None, None, :] + (w[None, :, :] - w[:, None, :])[None])  # R + t_n - t_m
        self.X = {k: t(v) for k, v in d['XX_R'].items()}

    def at(self, k):
        self.ph = torch.exp(2j * math.pi * (k @ self.R.T))
        self.E, self.U = torch.linalg.eigh(self._k(self.X['Ham']))
        dE = self.E[:, :, None] - self.E[:, None, :]
        self.dE, self.inv = dE, torch.where(dE.abs() < 1e-7, 0.0, 1.0 / dE)
        self.V = self.bar('Ham', 1)
        self.D = -self.V * self.inv[..., None]
        return self

    def _k(self, X):
        return (self.ph @ X.reshape(len(X), -1)).reshape((len(self.ph),) + X.shape[1:])

    def bar(self, key, der=0):
        X = self.X['AA'] if key == 'rotAA' else self.X[key]
        if key == 'rotAA':
            dX = self._der(X)
            X = dX[..., _BETA, _ALPHA] - dX[..., _ALPHA, _BETA]
        for _ in range(der):
            X = self._der(X)
        Xk = self._k(X).reshape(len(self.ph), self.nw, self.nw, -1).permute(0, 3, 1, 2)
        U = self.U[:, None]
        r = (U.mH @ Xk @ U).permute(0, 2, 3, 1)
        return r.reshape(r.shape[:3] + X.shape[3:])

    def _der(self, X):
        w = self.w.reshape(self.w.shape[:3] + (1,) * (X.dim() - 3) + (3,))
        return 1j * X[..., None] * w


def _mm(A, B):
    """[k, m, l, ...a] x [k, l, n, ...b] -> [k, m, n, a, b] summed over l."""
    a, b = A.shape[3:], B.shape[3:]
    r = torch.einsum('kmla,klnb->kmnab', A.reshape(A.shape[:3] + (-1,)), B.reshape(B.shape[:3] + (-1,)))
    return r.reshape(r.shape[:3] + a + b)


def _dn(A, B):
    """diagonal of A B: [k, n, l, a] x [k, l, n, a] -> [k, n, a] (component by component)."""
    return torch.einsum('knla,klna->kna', A, B)


def _omega(b):
    """Berry curvature per band [k, n, 3], all terms."""
    A, O, D = b.bar('AA'), b.bar('rotAA'), b.D
    s = 0.5 * torch.einsum('knnc->knc', O) - 1j * _dn(D[..., _ALPHA], D[..., _BETA])
    A0 = A * (1 - torch.eye(b.nw, device=A.device))[None, :, :, None]
    return 2 * (s - _dn(D[..., _ALPHA], A0[..., _BETA]) + _dn(D[..., _BETA], A0[..., _ALPHA])).real


def _derberry(b):
    """d_d Omega_c per band, [k, n, 3 (c), 3 (d)]."""
    V, W, D, A, dA, O, dO = b.V, b.bar('Ham', 2), b.D, b.bar('AA'), b.bar('AA', 1), b.bar('rotAA'), b.bar('rotAA', 1)
    sym = lambda t: t + t.transpose(3, 4)
    diag = lambda X: torch.einsum('knn...->kn...', X)
    Vd, Ad = diag(V), diag(A)
    dln = -b.inv[..., None, None] * (W + sym(_mm(V, D)) - sym(D[..., None] * Vd[:, None, :, None, :]))
    dnl = -b.inv[..., None, None] * (W + sym(Vd[:, :, None, :, None] * D[..., None, :]) - sym(_mm(D, V)))
    # group {n}: l, p run over the other bands (the diagonal of D is zero; of A it is taken out)
    dAln = dA - (D[..., None] * Ad[:, None, :, None, :]).transpose(3, 4) + _mm(A, D)
    dO_nn = diag(dO) - torch.einsum('knld,klnc->kncd', D, O) + torch.einsum('knlc,klnd->kncd', O, D)
    s = 0.5 * dO_nn.to(D.dtype)
    A0 = A * (1 - torch.eye(b.nw, device=A.device))[None, :, :, None]
    dAd = torch.einsum('knncd->kncd', dA) - torch.einsum('knld,klnc->kncd', D, A0) + torch.einsum('knlc,klnd->kncd', A0, D)
    pair = lambda X, Y: torch.einsum('knlc,klncd->kncd', X, Y)
    pair2 = lambda X, Y: torch.einsum('knlcd,klnc->kncd', X, Y)
    for sg, a, e in (1, _ALPHA, _BETA), (-1, _BETA, _ALPHA):
        s = s - 1j * sg * pair(D[..., a], dln[..., e, :]) - sg * pair(D[..., a], dAln[..., e, :])
        s = s - sg * pair2(dnl[..., a, :], A0[..., e]) - 1j * sg * Ad[..., a][..., None] * dAd[..., e, :]
    return 2 * s.real


def _morb(b):
    """H + G traces [k, n, 3] as differences of the sums over the n lowest bands (not additive), and Omega's."""
    D, A, B, C, E, O = b.D, b.bar('AA'), b.bar('BB'), b.bar('CC'), b.E, b.bar('rotAA')
    a, e = _ALPHA, _BETA
    El, En = E[:, None, :, None], E[:, :, None, None]  # energies of l (second index) and n (first) of the pair [k, n, l]
    T = lambda X: X.transpose(1, 2)
    dd = D[..., a] * T(D[..., e])
    pair = -1j * dd * (El + En) - D[..., a] * T(B[..., e]) + D[..., e] * T(B[..., a])
    pair = pair + En * (-D[..., a] * T(A[..., e]) + D[..., e] * T(A[..., a]))
    inner = -1j * A[..., a] * T(A[..., e]) * (El + En)  # pairs within the set
    single = 0.5 * torch.einsum('knnc->knc', C) + 0.5 * E[..., None] * torch.einsum('knnc->knc', O)
    cp, ci = pair.cumsum(1).cumsum(2), inner.cumsum(1).cumsum(2)
    d = lambda X: torch.einsum('knnc->knc', X)
    S = cp[:, :, -1] - d(cp) + d(ci) + single.cumsum(1)
    S = 2 * S.real
    return torch.cat([S[:, :1], S[:, 1:] - S[:, :-1]], 1)


def _scan(E, val, ef, fder):
    """Sum of per-band values over the states below each level; first central difference for fder 1."""
    dE = ef[1] - ef[0] if len(ef) > 1 else 0.001
    lo, n = ef[0] - fder * dE, len(ef) + 2 * fder
    i = torch.ceil((E - lo) / dE).clamp(min=0).to(torch.int64)
    i = torch.where(E > ef[-1] + fder * dE, n, i).reshape(-1)
    h = torch.zeros((n + 1,) + val.shape[2:], dtype=torch.float64, device=E.device)
    h.index_add_(0, i, val.reshape((-1,) + val.shape[2:]).double())
    h = h[:n].cumsum(0)
    return (h[2:] - h[:-2]) / (2 * dE) if fder else h


def _photo(b, ef, om, eta, sc_eta):
    V, W, D, A0, dA = b.V, b.bar('Ham', 2), b.D, b.bar('AA'), b.bar('AA', 1)
    A = A0 + 1j * D
    Dp = -V * (b.dE / (b.dE ** 2 + sc_eta ** 2))[..., None]
    diag = lambda X: torch.einsum('knn...->kn...', X)
    v, a = diag(V), diag(A0)
    row, col = (lambda x: x[:, :, None]), (lambda x: x[:, None, :])
    # [k, n, m, c, a]: a is the derivative's direction
    o = lambda x, y: x[..., :, None] * y[..., None, :]
    com = lambda X, x: (_mm(X, Dp) - _mm(Dp, X).transpose(3, 4) - o(row(x), Dp) + o(col(x), Dp))
    Ader = 1j * (W + com(V, v) + o(D, row(v) - col(v)) + o(row(v) - col(v), D)) * (-b.inv)[..., None, None]
    Ader = Ader + dA + com(A0, a) + o(D, row(a) - col(a)) + o(row(a) - col(a), D)
    Ader = Ader - 1j * o(A0, row(a) - col(a))
    M = -torch.einsum('knmca,kmnb->knmabc', Ader, A).imag
    M = M + M.transpose(4, 5)
    f = (b.E[..., None] <= ef).double()
    occ = f[:, None, :, :] - f[:, :, None, :]  # f(E_m) - f(E_n), levels last
    sel = occ.abs().amax(-1) > 0
    occ, M, x = occ[sel], M[sel].reshape(-1, 27), b.dE[sel][:, None]
    lor = lambda y: eta / math.pi / (y ** 2 + eta ** 2)
    fw = lor(x - om) + lor(-x - om)
    E1, E2 = b.E[:, :, None].expand(b.dE.shape)[sel][:, None], b.E[:, None, :].expand(b.dE.shape)[sel][:, None]
    keep = (x > om.min() - 5 * eta) & (x < om.max() + 5 * eta) & (E1 < ef.max()) & (E2 > ef.min())
    jd = torch.einsum('pe,pw->ew', occ, lor(x - om) * keep)
    return jd, torch.einsum('pw,pec->ewc', fw, occ[:, :, None] * M[:, None, :])


def _optical(b, ef, om, eta):
    A = b.bar('AA') + 1j * b.D
    f = (b.E[..., None] <= ef).double()
    occ = f[:, None, :, :] - f[:, :, None, :]
    sel = occ.abs().amax(-1) > 0
    M = (1j * A[..., :, None] * A.transpose(1, 2)[..., None, :])[sel].reshape(-1, 9)
    w = -b.dE[sel][:, None]  # E_m - E_n
    fw = w / (w - om - 1j * eta)
    r = fw.T @ (occ[sel][:, :, None] * M[:, None, :]).reshape(len(M), -1)
    return r.reshape(len(om), len(ef), 9).transpose(0, 1)


def exact(c, seed):
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    d = _model(c, seed)
    b = _Bands(d, dev)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=float)).to(dev)
    if c['kind'] == 'bands':
        b.at(t(np.random.default_rng(seed).uniform(0, 1, 3))[None])
        g = torch.einsum('knna->kna', b.V).real
        return {'energy': b.E[0].cpu().numpy(), 'band_gradients': g[0].cpu().numpy(),
                'berry_curvature': _omega(b)[0].cpu().numpy()}
    if c['tetra']:
        return None  # the tetrahedra's weights per k-point and level: minutes
    shifts, fft = _kgrid(c)
    j = np.stack(np.meshgrid(*[np.arange(n) for n in fft], indexing='ij'), -1).reshape(-1, 3)
    k = t(np.concatenate([j / fft + s for s in shifts]))
    ef, om = _axes(c)
    eft, omt = t(ef), t(om)
    step = max(1, min(len(k), int(6e8 / (c['nw'] ** 2 * 16 * {'dipole': 120, 'photo': 200, 'transport': 40,
                                                            'optical': 1 + c['nef'] * 8 + c['nomega']}.get(c['kind'], 20)))))
    acc, tab = {}, []

    def add(key, v):
        acc[key] = acc[key] + v if key in acc else v

    for i in range(0, len(k), step):
        b.at(k[i:i + step])
        if c['kind'] == 'tabulate':
            tab.append((b.E, torch.einsum('knna->kna', b.V).real, _omega(b)))
            continue
        if c['kind'] in ('ahc', 'dipole', 'optical'):
            add('ahc', _scan(b.E, _omega(b), ef, 0))
        if c['kind'] == 'dipole':
            add('dipole', _scan(b.E, _derberry(b), ef, 0))
        elif c['kind'] == 'optical':
            add('optical', _optical(b, eft, omt, 0.05))
        elif c['kind'] == 'photo':
            jd, sh = _photo(b, eft, omt, 0.05, 0.04)
            add('jdos', jd)
            add('shift', sh)
        elif c['kind'] == 'transport':
            v, o = torch.einsum('knna->kna', b.V).real, _omega(b)
            add('dos', _scan(b.E, torch.ones_like(b.E)[..., None], ef, 1))
            add('ohmic', _scan(b.E, v[..., :, None] * v[..., None, :], ef, 1))
            add('dipole', _scan(b.E, v[..., :, None] * o[..., None, :], ef, 1))
            add('morb', _scan(b.E, _morb(b), ef, 0) - 2 * eft[:, None] * _scan(b.E, o, ef, 0))
    if c['kind'] == 'tabulate':
        return {q: torch.cat(x).cpu().numpy() for q, x in zip(TAB, zip(*tab))}
    vol = abs(np.linalg.det(d['real_lattice']))
    nk = float(np.prod(fft)) * c['div'] ** 3
    scale = {'ahc': _AHC / vol, 'dipole': 1.0 / vol, 'optical': -_AHC / vol, 'jdos': 1.0 / vol, 'shift': _SHIFT / vol,
             'dos': 1.0, 'ohmic': _OHMIC / vol, 'morb': -1.0 / _HARTREE / _BOHR ** 2}
    out = {q: (v * (scale[q] / nk)).cpu().numpy() for q, v in acc.items()}
    if c['kind'] == 'dipole':
        out['dipole'] = out['dipole'].swapaxes(1, 2)
    for q, shape in (('dos', ()), ('jdos', None), ('optical', (3, 3)), ('shift', (3, 3, 3))):
        if q in out and shape is not None:
            out[q] = out[q].reshape((len(ef),) + ((len(om),) if q in ('optical', 'shift') else ()) + shape)
    return out
