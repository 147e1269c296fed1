"""A set-up issues all of its device work on its context's stream and ends with a wait for
it: builds run on non-blocking streams, which wait neither for that stream nor for the
legacy default stream, so a copy or clear left on either could land in the middle of a build.

On the CPU the sources of the set-up are read; on the GPU a set-up followed at once by a
build on a side stream runs while the legacy stream is held busy.  Tolerance 1e-11 of the
largest element: the order of the atomic sums.
"""
import os
import re

import pytest
import torch

from polymer_b200 import fock, geometry, inputdeck, scf, system

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'polymer_b200', 'csrc')


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return fh.read()


@pytest.mark.parametrize('name', ['pfe_mol.cu', 'pfe_lattice.cu', 'pfe_api.cu', 'pfe_eri.cu'])
def test_setup_sources_leave_nothing_on_the_legacy_stream(name):
    text = _source(name)
    if name == 'pfe_api.cu':
        text = text[text.index('static int setup_impl('):text.index('static int check_density(')]
        waits = text.rstrip().rsplit('cudaStreamSynchronize(s)', 1)
        assert len(waits) == 2 and 'alloc' not in waits[1] and 'cuda' not in waits[1]
    if name == 'pfe_eri.cu':
        text = text[text.index('int upload_optable('):text.index('int contract_outputs(')]
    assert re.findall(r'\bcuda(?:Memcpy|Memset)\([^;]*;', text) == []
    # kernel launches name their stream: four arguments between the brackets
    for launch in re.findall(r'<<<(.*?)>>>', text, flags=re.S):
        depth, commas = 0, 0
        for ch in launch:
            depth += ch in '({' or -(ch in ')}')
            commas += ch == ',' and depth == 0
        assert commas == 3, launch


@pytest.mark.gpu
@pytest.mark.parametrize('deck', [inputdeck.make_deck([1, 1], [[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]], 'STO-3G'),
                                  geometry.water_deck(1, 4), geometry.water_deck(3, 5)], ids=['H2', 'water', 'trimer'])
def test_build_right_after_setup_on_a_side_stream(deck):
    s = system.build_system(deck, fock.onee)
    p = torch.tensor(scf.guess_density(s)[0], dtype=torch.float64, device='cuda')
    first = fock.DeviceFock(s)
    ref = [t.clone() for t in first.from_pc(p)]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(5):
        torch.cuda._sleep(20_000_000)   # the legacy stream, some 10 ms
        with torch.cuda.stream(side):
            df = fock.DeviceFock(s)
            got = df.from_pc(p)
        side.synchronize()
        for g, r in zip(got, ref):
            assert float((g - r).abs().max()) <= 1e-11 * float(r.abs().max())
        df.close()
    first.close()
