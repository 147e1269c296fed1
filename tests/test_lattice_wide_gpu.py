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
from polymer_b200 import fock, inputdeck, scf, system

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
