"""Contexts of different molecules and chains alive at once: what a set-up does to a kernel
(its limit of dynamic shared memory is the kernel's, not the context's) must not change the
builds of another.  Each is built alone first; then all are set up, in both orders, and built
in turn, and then each from a thread of its own on a stream of its own.  Tolerance 1e-11 of
the largest element: the order of the atomic sums.
"""
import threading

import pytest
import torch

from polymer_b200 import fock, geometry, inputdeck, scf, system

pytestmark = pytest.mark.gpu

DECKS = {'ethane': geometry.alkane_deck(2), 'water': geometry.water_deck(1, 3), 'H2': inputdeck.make_deck(
    [1, 1], [[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]], 'STO-3G'),
    'dimer': geometry.water_deck(2, 4),
    'chain': geometry.polyethylene_deck('6-31Gss', cutoff1=1, cutoff2=1, kpoints=2, inttol=1e-8),
    'box': inputdeck.make_deck([8], [[0.1, 0.2, 0.3]], 'cc-pVDZ', period=(5.0, 5.5, 6.0), kpoints=(2, 2, 2), cutoff1=1,
                               cutoff2=1, inttol=1e-6)}


@pytest.fixture(scope='module')
def alone():
    out = {}
    for name, deck in DECKS.items():
        s = system.build_system(deck, fock.onee)
        b = s.basis
        pp = torch.tensor(b.cc.T @ scf.guess_density(s) @ b.cc, device='cuda')
        ph = scf.rotate(scf.HostState(s), pp.cpu())
        ph = ph.to('cuda') if ph is not None else None
        df = fock.DeviceFock(s)
        out[name] = (s, pp, ph, [t.clone() for t in df(pp, ph)])
        df.close()
    torch.cuda.synchronize()
    return out


def _worst(got, ref):
    return max(float((g - r).abs().max()) / float(r.abs().max()) for g, r in zip(got, ref))


@pytest.mark.parametrize('order', [1, -1])
def test_contexts_alive_at_once_build_as_alone(alone, order):
    names = list(alone)[::order]
    df = {n: fock.DeviceFock(alone[n][0]) for n in names}
    for n in names + names[::-1]:
        _, pp, ph, ref = alone[n]
        assert _worst(df[n](pp, ph), ref) <= 1e-11, n
    for d in df.values():
        d.close()


def test_contexts_of_several_threads_build_as_alone(alone):
    worst = {}

    def work(name):
        s, pp, ph, ref = alone[name]
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(6):
                df = fock.DeviceFock(s)
                for _ in range(2):
                    got = df(pp, ph)
                    stream.synchronize()
                    worst[name] = max(worst.get(name, 0.0), _worst(got, ref))
                df.close()

    threads = [threading.Thread(target=work, args=(n,)) for n in alone]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(worst) == sorted(alone)
    assert max(worst.values()) <= 1e-11, worst
