"""The digestion kernels of the straight-line molecular classes against the oracle for
every combination of kept shell components they are compiled for: p shells pure or with
an s component (sp), d shells pure or with lower components (shells that share one
exponent), and all quartet classes up to (22|22).  A build whose stored integrals exceed
one buffer runs in tiles (C20H42 in the full-size tests).

Tolerance as the other parity tests: 1e-11 of max|C_C| + 1e-13.
"""
import numpy as np
import pytest
import torch

import oracle
from polymer_b200 import fock, inputdeck, system

pytestmark = pytest.mark.gpu

# (typ, scale, [(exponent, coefficient[, p coefficient])]): the shells of one atom
BASES = {
    'pure p, pure d': [('S', 1.0, [(3.1, 0.4), (0.6, 0.7)]), ('P', 1.0, [(0.9, 1.0)]), ('D', 1.0, [(0.7, 1.0)])],
    'sp, pure d': [('S', 1.0, [(3.1, 1.0)]), ('SP', 1.0, [(1.4, 0.3, 0.5), (0.4, 0.8, 0.6)]), ('D', 1.0, [(0.7, 1.0)])],
    'pure p, spd': [('P', 1.0, [(1.3, 1.0)]), ('S', 1.0, [(0.6, 1.0)]), ('P', 1.0, [(0.6, 1.0)]), ('D', 1.0, [(0.6, 1.0)])],
    'sp, spd': [('SP', 1.0, [(1.3, 1.0, 0.8)]), ('S', 1.0, [(0.6, 1.0)]), ('P', 1.0, [(0.6, 1.0)]),
                ('D', 1.0, [(0.6, 1.0)])],
}


@pytest.mark.parametrize('name', sorted(BASES))
@pytest.mark.parametrize('primitive', [False, True])
def test_every_kept_combination_matches_the_oracle(name, primitive):
    deck = inputdeck.make_deck([1, 1, 1], [[0.0, 0.0, 0.0], [1.3, 0.2, -0.1], [-0.4, 1.1, 0.9]], '6-31G', inttol=1e-13)
    s = system.build_system(deck, oracle.onee, library={'H': BASES[name]})
    a = np.random.default_rng(5).normal(size=(s.basis.ncgs,) * 2) * 0.3
    pp = np.einsum('ai,cab,bj->cij', s.basis.cc, (a + a.T)[None], s.basis.cc, optimize=True)
    c_ref, x_ref = oracle.fourindex_eri(s, pp)
    df = fock.DeviceFock(s, primitive_targets=primitive)
    got = df(torch.tensor(pp, device='cuda'))
    torch.cuda.synchronize()
    for g, r in zip(got, (c_ref, x_ref)):
        assert np.abs(g.cpu().numpy() - r).max() <= 1e-11 * np.abs(r).max() + 1e-13
    df.close()
