"""Device memory that a context gives back: scratch of a set-up and of a call is cut again
for what follows, so calls at one geometry hold no more than the first of them, and a batch
holds what its molecules need.
"""
import ctypes

import numpy as np
import pytest
import torch

from polymer_b200 import capi, fock, geometry, system

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_gradient_calls_at_one_geometry_hold_no_more_than_the_first():
    """natom 5000 (all but three without a shell) makes the scratch of a call 240 KB."""
    L = capi.lib()
    s = system.build_system(geometry.water_deck(1, 3), fock.onee)
    pc = np.eye(s.basis.ncgs)
    pp = (s.basis.cc.T @ pc @ s.basis.cc)[None]
    a, keep = s.pfe_args(pp, None)
    natom = 5000
    atom = np.ascontiguousarray(s.basis.pgs_atom.astype(np.int32))
    out = []
    for k in range(150):
        gj, gk = np.zeros(3 * natom), np.zeros(3 * natom)
        capi.check(L, L.pfe_fourindex_eri_gradient(ctypes.byref(a), capi.iptr(atom), natom, capi.dptr(gj),
                                                   capi.dptr(gk)))
        if k in (1, 149):
            out.append((_free(), gj, gk))
    assert out[1][0] >= out[0][0]
    for i in (1, 2):
        assert np.abs(out[1][i] - out[0][i]).max() <= 1e-11 * np.abs(out[0][i]).max()


def test_batch_holds_what_its_molecules_need():
    """656 MiB on B200: up to 1.5 MiB of blocks a molecule and one buffer of stored integrals (1056 MiB where
    set-up scratch stays cut and every block is 2 MiB)."""
    s = system.build_system(geometry.water_deck(1, 3), fock.onee)
    fock.DeviceBatch([s, s]).close()   # modules and tables loaded
    before = _free()
    b = fock.DeviceBatch([s] * 256)
    held = before - _free()
    b.close()
    assert held <= 800 * MIB, held / MIB
