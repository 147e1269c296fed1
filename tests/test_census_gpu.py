"""The census's kernel_launches against the launches that the profiler sees in one build:
molecules (contracted and primitive targets, screening, classes in tiles, the ranks of a
build), lattices (straight-line, kept components, far cells, the interpreter alone), batches.
"""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from polymer_b200 import fock, geometry, inputdeck, scf, system

pytestmark = pytest.mark.gpu


def _launches(build):
    """Kernels of the library in one call of `build` (its names begin with the namespace)."""
    build()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
        build()
        torch.cuda.synchronize()
    return sum(1 for e in prof.events()
               if e.device_type == torch.autograd.DeviceType.CUDA and 'pfe::' in e.name)


def _primitive(sysm):
    b = sysm.basis
    return torch.tensor(b.cc.T @ scf.guess_density(sysm) @ b.cc, device='cuda')


MOLECULES = {
    'water': (geometry.water_deck(1, 3), {}, {}),
    'water, screened': (geometry.water_deck(1, 3), {}, dict(density_tol=1e-9)),
    'water, FP32': (geometry.water_deck(1, 3), {}, dict(mixed_cutoff=1e-6)),
    'butane, primitive targets': (geometry.alkane_deck(4), dict(primitive_targets=True), {}),
    'butane, rank 1 of 3': (geometry.alkane_deck(4), dict(myid=1, numprocs=3), {}),
    'C20H42, in tiles': (geometry.alkane_deck(20), {}, {}),
}


@pytest.mark.parametrize('name', sorted(MOLECULES))
def test_molecular_launches(name):
    deck, kw, screen = MOLECULES[name]
    s = system.build_system(deck, fock.onee)
    df = fock.DeviceFock(s, **kw)
    df.set_screening(**screen)
    pp = _primitive(s)
    assert df.census()['kernel_launches'] == _launches(lambda: df(pp))
    if not kw and not screen:
        df.force_variant(2)
        assert df.census()['kernel_launches'] == _launches(lambda: df(pp))
    df.close()


LATTICES = {
    'helix': geometry.polyethylene_deck('6-31Gss', cutoff1=1, cutoff2=2, kpoints=2, inttol=1e-8),
    'helix, no d': geometry.polyethylene_deck('STO-3G', cutoff1=1, cutoff2=2, kpoints=2, inttol=1e-8),
    'box': inputdeck.make_deck([6], [[0.1, 0.2, 0.3]], '6-31Gss', period=(5.0, 5.5, 6.0), kpoints=(2, 2, 2), cutoff1=1,
                               cutoff2=1, inttol=1e-6),
}


@pytest.mark.parametrize('name', sorted(LATTICES))
def test_lattice_launches(name):
    s = system.build_system(LATTICES[name], fock.onee)
    pp = _primitive(s)
    ph = scf.rotate(scf.HostState(s), pp.cpu())
    ph = ph.to('cuda') if ph is not None else None
    df = fock.DeviceFock(s)
    assert df.census()['kernel_launches'] == _launches(lambda: df(pp, ph))
    df.set_screening(mixed_cutoff=1e-6)
    assert df.census()['kernel_launches'] == _launches(lambda: df(pp, ph))
    df.set_screening()
    df.force_variant(1)
    assert df.census()['kernel_launches'] == _launches(lambda: df(pp, ph))
    df.close()


def test_batch_launches():
    systems = [system.build_system(d, fock.onee) for d in (geometry.water_deck(1, 3), geometry.alkane_deck(1))]
    b = fock.DeviceBatch(systems)
    for k, s in enumerate(systems):
        b.view(b.p_c, k).copy_(torch.tensor(scf.guess_density(s)[0], device='cuda'))
    assert b.census()['kernel_launches'] == _launches(lambda: b.run_packed(b.p_c, b.out_c, b.out_x))
    b.close()
