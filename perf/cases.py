"""The work that a user of this framework has it do, as measurable cases.

The framework's path is the direct two-electron Fock build of the polymer
Hartree-Fock code and what surrounds it on the device.  Each case is one pass
through a public entry point on a state that a user's program keeps:

* ``host``: ``fock.fourindex_eri``, the drop-in for FOURINDEX_ERI (host arrays
  in and out, static inputs cached in the library);
* ``device``: ``DeviceFock.__call__`` on a primitive density (molecules,
  chains, helices) of a context set up once;
* ``contracted``: ``DeviceFock.from_pc``, the SCF loop's form, plain, with the
  FP32 recursion of small quartets, or as an incremental build from a density
  difference with density screening;
* ``batch``: ``DeviceBatch.run_packed``, many molecules of uneven size at once;
* ``gradient``: ``fock.fourindex_eri_gradient``, the two-electron gradient;
* ``onee``: ``fock.onee``, the one-electron integrals of a new geometry.

The systems are those of the repository's configurations and tests: the water
single point and water clusters in cc-pVDZ, all-trans alkanes in 6-31G**, and
helical polyethylene.  The geometry carries seeded jitter (or seeded placement),
the density is the nuclear-charge diagonal plus seeded off-diagonal elements
that decay with distance, as a converged density's do.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from polymer_b200 import fock, geometry, inputdeck, system

F64 = torch.float64


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one water molecule through the Fortran-facing call: the smallest build, host call overhead and launches
        dict(name='water_host', entry='host', kind='water', size=1, inttol=1e-12),
        # the same molecule inside a device SCF loop: launches and latency
        dict(name='water_scf', entry='contracted', kind='water', size=1, inttol=1e-12),
        # a small molecule's build from the primitive density
        dict(name='butane', entry='device', kind='alkane', size=4, inttol=1e-10),
        # an ordinary molecule in the SCF loop
        dict(name='decane_scf', entry='contracted', kind='alkane', size=10, inttol=1e-10),
        # the mixed-precision option on it
        dict(name='decane_mixed', entry='contracted', kind='alkane', size=10, inttol=1e-10, mixed=1e-6),
        # the build benchmark: a large molecule, full build
        dict(name='eicosane', entry='device', kind='alkane', size=20, inttol=1e-10),
        # a later SCF iteration of it: incremental build with density screening
        dict(name='eicosane_incremental', entry='contracted', kind='alkane', size=20, inttol=1e-10, dtol=1e-8,
             delta=1e-4),
        # many clusters of uneven size in one build: the largest case
        dict(name='water_batch', entry='batch', kind='water', size=16, count=12, inttol=1e-10),
        # helical polymer, the lattice path without d shells, at its configured cutoffs
        dict(name='helix_631g', entry='device', kind='helix', basis='6-31G', size=5, cutoff2=10, inttol=1e-10),
        # the same chain with polarisation functions, smaller cutoffs
        dict(name='helix_631gss', entry='device', kind='helix', basis='6-31Gss', size=1, cutoff2=2, inttol=1e-10),
        # forces of a geometry step
        dict(name='gradient_ethane', entry='gradient', kind='alkane', size=2, inttol=1e-10),
        # the one-electron integrals of a geometry step
        dict(name='onee_decane', entry='onee', kind='alkane', size=10, inttol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges."""
    entry = rng.choice(['host', 'device', 'contracted', 'contracted', 'batch', 'helix', 'gradient', 'onee'])
    inttol = rng.choice([1e-9, 1e-10, 1e-11, 1e-12])
    if entry == 'helix':
        c1 = rng.randint(1, 5)
        return dict(entry='device', kind='helix', basis=rng.choice(['STO-3G', '6-31G']), size=c1,
                    cutoff2=rng.randint(c1, 2 * c1), inttol=max(inttol, 1e-10))
    if entry == 'batch':
        return dict(entry='batch', kind='water', size=_log_int(rng, 1, 14), count=_log_int(rng, 2, 10),
                    inttol=max(inttol, 1e-10))
    if entry == 'gradient':
        kind = rng.choice(['alkane', 'water'])
        return dict(entry=entry, kind=kind, size=_log_int(rng, 1, 2), inttol=inttol)
    kind = rng.choice(['alkane', 'water'])
    case = dict(entry=entry, kind=kind, size=_log_int(rng, 1, 17 if kind == 'alkane' else 10), inttol=inttol)
    if entry == 'contracted':
        option = rng.choice(['plain', 'mixed', 'incremental'])
        if option == 'mixed':
            case['mixed'] = rng.choice([1e-7, 1e-6, 1e-5])
        elif option == 'incremental':
            case['delta'] = rng.choice([1e-5, 1e-4, 1e-3])
            case['dtol'] = min(max(1e-11, 1e-4 * case['delta']), 1e-8)
    return case


# ------------------------------------------------------------------ states

def _decks(case, seed):
    kind, size, opts = case['kind'], case['size'], dict(inttol=case['inttol'])
    if kind == 'alkane':
        atoms, xyz = geometry.alkane(size, seed=seed)
        return [inputdeck.make_deck(atoms, xyz, '6-31Gss', **opts)]
    if kind == 'helix':
        return [geometry.polyethylene_deck(case['basis'], cutoff1=size, cutoff2=case['cutoff2'], kpoints=4, seed=seed,
                                           **opts)]
    opts['spherical'] = True
    if case['entry'] != 'batch':
        return [geometry.water_deck(size, seed, **opts)]
    # cluster sizes evenly over 1..size, the same for every seed, so that a case is one amount of work
    n = case['count']
    sizes = [max(1, round(1 + (size - 1) * (k + 0.5) / n)) for k in range(n)]
    return [geometry.water_deck(k, 1000 * seed + i, **opts) for i, k in enumerate(sizes)]


def _density(sysm, seed, delta=0.0):
    """A symmetric contracted density, cell-major: the nuclear-charge diagonal and
    decaying off-diagonal elements; with `delta` a density difference of that size."""
    rng = np.random.default_rng(seed)
    b, n, nc = sysm.basis, sysm.basis.ncgs, sysm.ncell1
    d = np.linalg.norm(b.cgs[:, None] - b.cgs[None], axis=-1)
    period = np.array(sysm.deck.period)
    p = np.zeros((nc, n, n))
    for c, q in enumerate(sysm.cells):
        m = sysm.cell_index(-q[0], -q[1], -q[2])
        if m < c:
            p[c] = p[m].T           # P(-q) = P(q)^T
            continue
        far = np.linalg.norm(np.array(q) * period)
        a = rng.normal(size=(n, n)) * np.exp(-0.5 * (d + far))
        p[c] = a if m != c else 0.5 * (a + a.T)
    if delta:
        return delta * p
    p *= 0.3
    real = np.any(b.cc != 0.0, axis=1)
    c0 = sysm.cell_index(0, 0, 0)
    for k in np.nonzero(real)[0]:
        atom = int(np.argmin(np.linalg.norm(np.array(sysm.deck.coords) - b.cgs[k], axis=1)))
        p[c0, k, k] += sysm.deck.atoms[atom] / (1.0 + float(np.sum(real & (d[k] == 0.0))))
    return p


def _rotated(sysm, pp):
    """P_P_HELIX of a primitive density (ROTATE_DENSITYMATRIX), on the host."""
    c1, c2 = sysm.deck.cel1[0], sysm.deck.cel2[0]
    h = c1 + c2
    out = np.zeros((2 * h + 1, 2 * c2 + 1) + pp.shape[1:])
    for q2 in range(-c2, c2 + 1):
        for q1 in range(max(-h, q2 - c1), min(h, q2 + c1) + 1):
            out[q1 + h, q2 + c2] = sysm.p2h[q2 + h].T @ pp[sysm.cell_index(q1 - q2)] @ sysm.p2h[q1 + h]
    return out


def prepare(case, seed):
    entry, dev = case['entry'], torch.device('cuda')
    decks = _decks(case, seed)
    systems = [system.build_system(d, fock.onee) for d in decks]
    s = systems[0]
    if entry == 'onee':
        return dict(entry=entry, system=s)
    pcs = [_density(m, seed + 17 * k, case.get('delta', 0.0)) for k, m in enumerate(systems)]
    if entry == 'batch':
        fb = fock.DeviceBatch(systems)
        for k, p in enumerate(pcs):
            fb.view(fb.p_c, k).copy_(torch.tensor(p[0], device=dev))
        return dict(entry=entry, system=s, fock=fb)
    pc, cc = pcs[0], s.basis.cc
    pp = cc.T @ pc @ cc
    if entry in ('host', 'gradient'):
        return dict(entry=entry, system=s, p=pp)
    state = dict(entry=entry, system=s)
    if entry == 'contracted':
        state['fock'] = fock.DeviceFock(s)
        if 'mixed' in case or 'dtol' in case:
            state['fock'].set_screening(case.get('mixed', 0.0), case.get('dtol', 0.0))
        state['p'] = torch.tensor(pc, device=dev)
    else:
        state['fock'] = fock.DeviceFock(s)
        state['p'] = torch.tensor(pp, device=dev)
        state['ph'] = torch.tensor(_rotated(s, pp), device=dev) if s.deck.helix != 0.0 else None
    return state


def run(state):
    entry = state['entry']
    if entry == 'host':
        return fock.fourindex_eri(state['system'], state['p'])
    if entry == 'gradient':
        return fock.fourindex_eri_gradient(state['system'], state['p'])
    if entry == 'onee':
        return fock.onee(state['system'])
    fk = state['fock']
    if entry == 'batch':
        fk.run_packed(fk.p_c, fk.out_c, fk.out_x)
        return fk.out_c, fk.out_x
    if entry == 'contracted':
        return fk.from_pc(state['p'])
    return fk(state['p'], state['ph'])


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Each input matrix read and each output matrix written once.  The operations
    are those of the quartets that pass the screen, one recursion each, as the
    library's census counts them (the gradient: nine derivative integrals for
    each); the one-electron integrals: about 60 per primitive pair and nucleus."""
    systems = [system.build_system(d, fock.onee) for d in _decks(case, 1)]
    if case['entry'] == 'onee':
        n2 = float(systems[0].basis.npgs) ** 2
        return {'bytes': 3 * 8 * n2, 'flops': 60.0 * n2 * systems[0].deck.natom}
    if case['entry'] == 'batch':
        fk = fock.DeviceBatch(systems)
        bytes_ = 3 * 8.0 * fk.off[-1]
    else:
        fk = fock.DeviceFock(systems[0])
        b, nc = systems[0].basis, systems[0].ncell1
        np_ = b.ncgs if case['entry'] == 'contracted' else b.npgs
        bytes_ = 8.0 * nc * (np_ ** 2 + 2 * b.ncgs ** 2)
    flops = fk.census()['flops']
    fk.close()
    return {'bytes': bytes_, 'flops': (9.0 if case['entry'] == 'gradient' else 1.0) * flops}


def tolerance(case):
    """FP64 throughout: sums in another order and the Boys function to its table's
    accuracy (about 1e-14).  The mixed option moves every quartet near its cutoff
    by an FP32 rounding; which quartets take FP32 follows the order of the work."""
    if 'mixed' in case:
        return {'rel': 1e-8, 'max': 1e-6}
    return {'rel': 1e-11, 'max': 1e-9}


# ------------------------------------------------------------------ the same in plain FP64 tensor operations

_PI = 3.14159265358979   # the constant the method is defined with


def _boys(n, t):
    """F_0..F_n(t): the ascending series below 40 (downward recursion), the asymptotic form above."""
    lo = torch.clamp(t, max=40.0)
    term = torch.full_like(lo, 1.0 / (2 * n + 1))
    top = term.clone()
    for k in range(1, 180):
        term = term * (2.0 * lo / (2 * n + 2 * k + 1))
        top = top + term
    e = torch.exp(-lo)
    f = [None] * (n + 1)
    f[n] = e * top
    for m in range(n, 0, -1):
        f[m - 1] = (2.0 * lo * f[m] + e) / (2 * m - 1)
    big, v = t > 40.0, 0.5 * torch.sqrt(_PI / torch.clamp(t, min=40.0))
    for m in range(n + 1):
        f[m] = torch.where(big, v, f[m])
        v = v * (2 * m + 1) / (2.0 * torch.clamp(t, min=40.0))
    return f


def _hermite_1d(i, j, t, a, b, ab):
    """Hermite expansion coefficient E_t^{ij} of x_A^i x_B^j (overlap factor left out)."""
    p = a + b
    if t < 0 or t > i + j:
        return torch.zeros_like(p)
    if i == j == 0:
        return torch.ones_like(p)
    if i > 0:
        pa = -b / p * ab
        return (_hermite_1d(i - 1, j, t - 1, a, b, ab) / (2 * p) + pa * _hermite_1d(i - 1, j, t, a, b, ab)
                + (t + 1) * _hermite_1d(i - 1, j, t + 1, a, b, ab))
    pb = a / p * ab
    return (_hermite_1d(i, j - 1, t - 1, a, b, ab) / (2 * p) + pb * _hermite_1d(i, j - 1, t, a, b, ab)
            + (t + 1) * _hermite_1d(i, j - 1, t + 1, a, b, ab))


def _hermites(n):
    return [(x, y, z) for x in range(n + 1) for y in range(n + 1 - x) for z in range(n + 1 - x - y)]


def _coulomb(alpha, d, n):
    """Hermite Coulomb integrals R_{xyz}(alpha, d) with x + y + z <= n."""
    f = _boys(n, alpha * (d * d).sum(-1))
    r = {(0, 0, 0, m): (-2.0 * alpha) ** m * f[m] for m in range(n + 1)}
    for h in sorted(_hermites(n), key=sum)[1:]:
        i = next(k for k in range(3) if h[k])
        h1 = tuple(v - (k == i) for k, v in enumerate(h))
        h2 = tuple(v - 2 * (k == i) for k, v in enumerate(h))
        for m in range(n + 1 - sum(h)):
            v = d[..., i] * r[h1 + (m + 1,)]
            r[h + (m,)] = v + h1[i] * r[h2 + (m + 1,)] if h1[i] else v
    return {h: r[h + (0,)] for h in _hermites(n)}


class _Pairs:
    """The Hermite expansion of every product of two primitives, by distinct
    (exponent, centre) pair."""

    def __init__(self, b, xyz):
        dev = xyz.device
        key = {}
        self.shell = [key.setdefault((int(a), float(z)), len(key)) for a, z in zip(b.pgs_atom, b.zt)]
        zeta = torch.tensor([k[1] for k in key], device=dev, dtype=F64)
        at = xyz[torch.tensor([k[0] - 1 for k in key], device=dev)]
        self.a, self.b = zeta[:, None].expand(len(key), len(key)), zeta[None, :].expand(len(key), len(key))
        self.p = self.a + self.b
        self.ab = at[:, None] - at[None]
        self.centre = (self.a[..., None] * at[:, None] + self.b[..., None] * at[None]) / self.p[..., None]
        self.overlap = torch.exp(-self.a * self.b / self.p * (self.ab ** 2).sum(-1)) * (_PI / self.p) ** 1.5
        self.index = torch.tensor(self.shell, device=dev)
        self.powers = [(int(x), int(y), int(z)) for x, y, z in zip(b.pax, b.pay, b.paz)]
        self.herm = _hermites(4)
        self.ns = len(key)
        memo = {}

        def e1(i, j, t, k):
            if (i, j, t, k) not in memo:
                memo[i, j, t, k] = _hermite_1d(i, j, t, self.a, self.b, self.ab[..., k])
            return memo[i, j, t, k]

        self.e1 = e1

    def fold(self, weight):
        """sum over primitive pairs of weight[..., i, j] E^{ij}_h -> [..., shell, shell, h]."""
        lead = weight.shape[:-2]
        parts = []
        by_power = {}
        for i, pw in enumerate(self.powers):
            by_power.setdefault(pw, []).append(i)
        w = {}
        for pa, ia in by_power.items():
            for pb, ib in by_power.items():
                sub = weight[..., ia, :][..., :, ib]
                ra = torch.zeros((len(ia), self.ns), dtype=F64, device=weight.device)
                rb = torch.zeros((len(ib), self.ns), dtype=F64, device=weight.device)
                ra[torch.arange(len(ia)), self.index[ia]] = 1.0
                rb[torch.arange(len(ib)), self.index[ib]] = 1.0
                w[pa, pb] = ra.T @ sub @ rb
        for h in self.herm:
            tot = torch.zeros(lead + (self.ns, self.ns), dtype=F64, device=weight.device)
            for (pa, pb), v in w.items():
                if all(h[k] <= pa[k] + pb[k] for k in range(3)):
                    tot = tot + v * (self.e1(pa[0], pb[0], h[0], 0) * self.e1(pa[1], pb[1], h[1], 1)
                                     * self.e1(pa[2], pb[2], h[2], 2))
            parts.append(tot)
        return torch.stack(parts, -1) * self.overlap[..., None]


def _repulsion_blocks(pr, rows=64):
    """(first pair, T) over blocks of shell pairs: T[p, q, h, g] = 2 sqrt(rho/pi) (-1)^|g| R_{h+g}."""
    p, c = pr.p.reshape(-1), pr.centre.reshape(-1, 3)
    herm = pr.herm
    sign = torch.tensor([(-1.0) ** sum(g) for g in herm], dtype=F64, device=p.device)
    for k in range(0, p.numel(), rows):
        alpha = p[k:k + rows, None] * p[None] / (p[k:k + rows, None] + p[None])
        r = _coulomb(alpha, c[k:k + rows, None] - c[None], 8)
        pref = 2.0 * torch.sqrt(alpha / _PI)
        t = torch.stack([torch.stack([r[tuple(u + v for u, v in zip(h, g))] for g in herm], -1) for h in herm], -2)
        yield k, t * pref[..., None, None] * sign


def _integrals(b, xyz):
    """(ij|kl) over the contracted functions that carry a coefficient, and their rows."""
    rows = np.nonzero(np.any(b.cc != 0.0, axis=1))[0]
    pr = _Pairs(b, xyz)
    cc = torch.tensor(b.cc[rows], device=xyz.device)
    n = len(rows)
    i, j = np.tril_indices(n)
    pairs = pr.fold(cc[i][:, :, None] * cc[j][:, None, :]).reshape(len(i), pr.ns ** 2, -1)
    out = torch.zeros(len(i), len(i), dtype=F64, device=xyz.device)
    flat = pairs.reshape(len(i), -1)
    for k, t in _repulsion_blocks(pr):
        m = t.shape[0]
        bra = pairs[:, k:k + m]
        for s in range(m):
            live = bra[:, s].abs().amax(-1) > 0.0
            pot = torch.einsum('qhg->hqg', t[s]).reshape(len(pr.herm), -1)
            out[live] += bra[live, s] @ (pot @ flat.T)
    full = torch.zeros(n, n, len(i), dtype=F64, device=xyz.device)
    full[i, j] = out
    full[j, i] = out
    eri = torch.zeros(n, n, n, n, dtype=F64, device=xyz.device)
    eri[:, :, i, j] = full
    eri[:, :, j, i] = full
    return eri, rows


def exact(case, seed):
    """One water molecule's J and K from all of its integrals by the
    McMurchie-Davidson scheme; larger systems take too long this way."""
    if case['kind'] != 'water' or case['size'] != 1 or case['entry'] not in ('host', 'contracted', 'device') \
            or 'mixed' in case or 'dtol' in case:
        return None
    s = system.build_system(_decks(case, seed)[0], fock.onee)
    dev = torch.device('cuda')
    eri, rows = _integrals(s.basis, torch.tensor(np.array(s.deck.coords), device=dev, dtype=F64))
    p = torch.tensor(_density(s, seed, case.get('delta', 0.0))[0][np.ix_(rows, rows)], device=dev)
    n = s.basis.ncgs
    c, x = (torch.zeros(1, n, n, dtype=F64, device=dev) for _ in range(2))
    at = torch.tensor(rows, device=dev)
    c[0, at[:, None], at[None]] = torch.einsum('ijkl,kl->ij', eri, p)
    x[0, at[:, None], at[None]] = torch.einsum('ikjl,kl->ij', eri, p)
    return (c.cpu().numpy(), x.cpu().numpy()) if case['entry'] == 'host' else (c, x)
