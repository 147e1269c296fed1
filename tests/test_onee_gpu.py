"""Nuclear attraction integrals per class of shell pairs (both orders of unequal classes,
cells, helix images, every d shell kind) against the oracle: 1e-12 of the largest element,
which covers the two recursions' rounding over a few hundred operations.
"""
import numpy as np
import pytest

import oracle
from polymer_b200 import fock, geometry, inputdeck, system

pytestmark = pytest.mark.gpu

ONE = inputdeck.make_deck([1], [[0.1, 0.2, 0.3]], 'STO-3G', inttol=0.0)
DECKS = {'one shell': ONE, 'water': geometry.water_deck(1, 3), 'ethane': geometry.alkane_deck(2),
         'helix with d': geometry.polyethylene_deck('6-31Gss', cutoff1=1, cutoff2=2, kpoints=2),
         'box': inputdeck.make_deck([6], [[0.1, 0.2, 0.3]], '6-31Gss', period=(5.0, 5.5, 6.0), kpoints=(2, 2, 2),
                                    cutoff1=1, cutoff2=1, inttol=1e-10)}


@pytest.mark.parametrize('name', sorted(DECKS))
def test_one_electron_integrals_match_the_oracle(name):
    s = system.build_system(DECKS[name], oracle.onee)
    for got, ref in zip(fock.onee(s), (s.s_p, s.t_p, s.n_p)):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max() + 1e-14
