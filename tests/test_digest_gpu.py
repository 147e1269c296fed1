"""The digestion kernels of the straight-line molecular classes against the oracle for
every combination of kept shell components they are compiled for: p shells pure or with
an s component (sp), d shells pure or with lower components (shells that share one
exponent), and all quartet classes up to (22|22); a batch that joins all four; and, with the
memory for stored integrals cut to a few chunks, builds whose classes run in many tiles (the
last of them partly filled), for one rank, for three, and for a batch.

Tolerance as the other parity tests: 1e-11 of max|C_C| + 1e-13.
"""
import numpy as np
import pytest
import torch

import oracle
from polymer_b200 import capi, fock, geometry, inputdeck, system

pytestmark = pytest.mark.gpu

# (typ, scale, [(exponent, coefficient[, p coefficient])]): the shells of one atom
BASES = {
    'pure p, pure d': [('S', 1.0, [(3.1, 0.4), (0.6, 0.7)]), ('P', 1.0, [(0.9, 1.0)]), ('D', 1.0, [(0.7, 1.0)])],
    'sp, pure d': [('S', 1.0, [(3.1, 1.0)]), ('SP', 1.0, [(1.4, 0.3, 0.5), (0.4, 0.8, 0.6)]), ('D', 1.0, [(0.7, 1.0)])],
    'pure p, spd': [('P', 1.0, [(1.3, 1.0)]), ('S', 1.0, [(0.6, 1.0)]), ('P', 1.0, [(0.6, 1.0)]), ('D', 1.0, [(0.6, 1.0)])],
    'sp, spd': [('SP', 1.0, [(1.3, 1.0, 0.8)]), ('S', 1.0, [(0.6, 1.0)]), ('P', 1.0, [(0.6, 1.0)]),
                ('D', 1.0, [(0.6, 1.0)])],
}


def _case(s, seed):
    """A system, a contracted density, its decontraction and the oracle's J and K."""
    a = np.random.default_rng(seed).normal(size=(s.basis.ncgs,) * 2) * 0.3
    pp = np.einsum('ai,cab,bj->cij', s.basis.cc, (a + a.T)[None], s.basis.cc, optimize=True)
    return s, a + a.T, pp, oracle.fourindex_eri(s, pp)


def _basis_case(name, seed=5):
    deck = inputdeck.make_deck([1, 1, 1], [[0.0, 0.0, 0.0], [1.3, 0.2, -0.1], [-0.4, 1.1, 0.9]], '6-31G', inttol=1e-13)
    return _case(system.build_system(deck, oracle.onee, library={'H': BASES[name]}), seed)


def _close(got, ref):
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max() + 1e-13


@pytest.mark.parametrize('name', sorted(BASES))
@pytest.mark.parametrize('primitive', [False, True])
def test_every_kept_combination_matches_the_oracle(name, primitive):
    s, _, pp, ref = _basis_case(name)
    df = fock.DeviceFock(s, primitive_targets=primitive)
    got = df(torch.tensor(pp, device='cuda'))
    torch.cuda.synchronize()
    for g, r in zip(got, ref):
        _close(g.cpu().numpy(), r)
    df.close()


@pytest.mark.parametrize('order', [1, -1])
def test_batch_of_all_kept_combinations_matches_the_oracle(order):
    """Molecules of pure d shells and of d shells with lower components share launches and panels that keep what
    any of them needs, in either order (the joined launches begin as copies of the first one's)."""
    cases = [_basis_case(n, 6 + k) for k, n in enumerate(sorted(BASES))][::order]
    b = fock.DeviceBatch([c[0] for c in cases])
    got = b([torch.tensor(c[1], device='cuda') for c in cases])
    torch.cuda.synchronize()
    for (_, _, _, ref), g in zip(cases, got):
        for k in range(2):
            _close(g[k].cpu().numpy(), ref[k][0])
    b.close()


@pytest.fixture
def small_tiles():
    """Set-ups with 128 KiB for a class's stored integrals (a chunk of (21|21) is 83 KB of pure shells, one of
    (10|00) 768 bytes) and no classes side by side."""
    L = capi.lib()
    L.pfe_debug_integral_memory(128 << 10, 1)
    yield
    L.pfe_debug_integral_memory(0, 0)


TILED = {'dimer': geometry.water_deck(2, 16, inttol=1e-12), 'methane': geometry.alkane_deck(1, inttol=1e-12)}


@pytest.mark.parametrize('name', sorted(TILED))
@pytest.mark.parametrize('ranks', [1, 3])
def test_tiles_match_the_oracle(small_tiles, name, ranks):
    s, _, pp, ref = _case(system.build_system(TILED[name], oracle.onee), 9)
    d = torch.tensor(pp, device='cuda')
    total = [0.0, 0.0]
    for r in range(ranks):
        df = fock.DeviceFock(s, myid=r, numprocs=ranks)
        capi.lib().pfe_debug_integral_memory(0, 0)
        whole = fock.DeviceFock(s, myid=r, numprocs=ranks)
        capi.lib().pfe_debug_integral_memory(128 << 10, 1)
        # several tiles in several classes: a tile adds the launches of its class again
        assert df.census()['kernel_launches'] >= 2 * whole.census()['kernel_launches']
        for rep in range(2):   # a second build on what the first left behind
            got = [g.cpu().numpy() for g in df(d)]
        total = [t + g for t, g in zip(total, got)]
        for x in (df, whole):
            x.close()
    for t, r in zip(total, ref):
        _close(t, r)


def test_tiles_of_a_batch_match_the_oracle(small_tiles):
    cases = [_case(system.build_system(d, oracle.onee), 11 + k) for k, d in
             enumerate([geometry.water_deck(1, 17, inttol=1e-12), geometry.alkane_deck(1, inttol=1e-12)])]
    b = fock.DeviceBatch([c[0] for c in cases])
    capi.lib().pfe_debug_integral_memory(0, 0)
    whole = fock.DeviceBatch([c[0] for c in cases])
    assert b.census()['kernel_launches'] >= 2 * whole.census()['kernel_launches']
    whole.close()
    for rep in range(2):
        got = b([torch.tensor(c[1], device='cuda') for c in cases])
    torch.cuda.synchronize()
    for (_, _, _, ref), g in zip(cases, got):
        for k in range(2):
            _close(g[k].cpu().numpy(), ref[k][0])
    b.close()
