"""Lattice and helix builds with d shells against the oracle: the kernels that keep the
top-level components of pure d shells (either order of bra and ket class), the interpreter
they leave a build to when some ghost carries density, and bases whose d shells keep their
lower components, which never take them.

Tolerance as the other lattice tests: 1e-11 of max|C_C| + 1e-13.
"""
import numpy as np
import pytest
import torch

import oracle
from polymer_b200 import fock, geometry, inputdeck, scf, system

pytestmark = pytest.mark.gpu

PURE = [('SP', 1.0, [(1.1, 0.6, 0.7)]), ('P', 1.0, [(0.8, 1.0)]), ('D', 1.0, [(0.9, 1.0)])]
LOWER = [('S', 1.0, [(0.9, 1.0)]), ('P', 1.0, [(0.9, 1.0)]), ('D', 1.0, [(0.9, 1.0)]), ('P', 1.0, [(0.5, 1.0)])]


@pytest.mark.parametrize('ghosts', [False, True])
@pytest.mark.parametrize('helix', [0.0, 40.0])
@pytest.mark.parametrize('shells', [PURE, LOWER], ids=['pure', 'lower'])
def test_d_shells_match_the_oracle(shells, helix, ghosts):
    deck = inputdeck.make_deck([1, 1], [[0.0, 0.3, 0.1], [1.5, -0.2, 0.4]], '6-31G', period=(4.5, 0.0, 0.0),
                               helix_deg=helix, kpoints=(2, 0, 0), cutoff1=1, cutoff2=1, inttol=1e-11)
    s = system.build_system(deck, oracle.onee, library={'H': shells})
    rng = np.random.default_rng(3)
    n = s.basis.ncgs
    pc = rng.normal(size=(s.ncell1, n, n)) * 0.2
    for c, q in enumerate(s.cells):
        m = s.cell_index(-q[0], -q[1], -q[2])
        if m <= c:
            pc[c] = pc[m].T if m < c else 0.5 * (pc[c] + pc[c].T)
    pp = np.einsum('ai,cab,bj->cij', s.basis.cc, pc, s.basis.cc, optimize=True)
    if ghosts:   # not a decontracted density: every primitive carries some
        pp = pp + 0.05 * rng.normal(size=pp.shape)
    ph = scf.rotate(scf.HostState(s), torch.tensor(pp))
    ph = ph.numpy() if ph is not None else None
    ref = oracle.fourindex_eri(s, pp, ph)
    got = fock.fourindex_eri(s, pp, ph)
    for g, r in zip(got, ref):
        assert np.abs(g - r).max() <= 1e-11 * np.abs(ref[0]).max() + 1e-13


def test_builds_with_ghost_densities_are_no_slower_than_the_interpreter_alone():
    """Where ghosts carry density the d classes fall back to the interpreter.  With the far-cell cutoff set and no
    cell outside the CUTOFF1 box the same kernels do the same FP64 work without the attempt before them: the
    fallback may cost its empty launches and the check (here some 2 %), no more."""
    deck = geometry.polyethylene_deck('6-31Gss', cutoff1=1, cutoff2=1, kpoints=2, inttol=1e-10)
    s = system.build_system(deck, fock.onee)
    rng = np.random.default_rng(4)
    pp = torch.tensor(0.05 * rng.normal(size=(s.ncell1, s.basis.npgs, s.basis.npgs)), device='cuda')
    ph = scf.rotate(scf.HostState(s), pp.cpu()).to('cuda')
    df = fock.DeviceFock(s)

    def best():
        times = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            out = df(pp, ph)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times), out

    fallback, a = best()
    df.set_screening(mixed_cutoff=1e-30)
    alone, b = best()
    df.close()
    for x, y in zip(a, b):
        assert float((x - y).abs().max()) <= 1e-11 * float(b[0].abs().max())
    assert fallback <= 1.05 * alone, (fallback, alone)
