"""Chunks cut into pieces (small molecules: their long contractions make lanes
that walk thousands of primitive quartets) against the oracle: whole builds, the
rank split over the cut lists, and a batch whose pieces carry their instance.

Tolerance as the other parity tests: 1e-11 of max|C_C| + 1e-13.
"""
import numpy as np
import pytest
import torch

import oracle
from polymer_b200 import fock, geometry, system

pytestmark = pytest.mark.gpu


def _case(deck, seed):
    s = system.build_system(deck, oracle.onee)
    a = np.random.default_rng(seed).normal(size=(s.basis.ncgs,) * 2) * 0.3
    pc = a + a.T
    pp = np.einsum('ai,cab,bj->cij', s.basis.cc, pc[None], s.basis.cc, optimize=True)
    return s, pc, pp, oracle.fourindex_eri(s, pp)


def _close(got, ref):
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max() + 1e-13


@pytest.mark.parametrize('ranks', [1, 3])
@pytest.mark.parametrize('deck', [geometry.water_deck(1, 5, inttol=0.0), geometry.water_deck(2, 6, inttol=1e-12),
                                  geometry.alkane_deck(1, inttol=1e-12)], ids=['water', 'dimer', 'methane'])
def test_cut_chunks_match_the_oracle(deck, ranks):
    s, _, pp, ref = _case(deck, 3)
    parts = [fock.fourindex_eri(s, pp, myid=r, numprocs=ranks) for r in range(ranks)]
    for k in range(2):
        _close(sum(p[k] for p in parts), ref[k])


def test_cut_chunks_of_a_batch_match_the_oracle():
    cases = [_case(geometry.water_deck(1, 8, inttol=1e-12), 1), _case(geometry.alkane_deck(1, inttol=1e-12), 2),
             _case(geometry.water_deck(2, 9, inttol=1e-12), 4)]
    b = fock.DeviceBatch([c[0] for c in cases])
    got = b([torch.tensor(c[1], device='cuda') for c in cases])
    torch.cuda.synchronize()
    for (_, _, _, ref), g in zip(cases, got):
        for k in range(2):
            _close(g[k].cpu().numpy(), ref[k][0])
    b.close()
