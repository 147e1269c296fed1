"""Error paths of the set-up under injected device-allocation failures
(pfe_debug_fail_allocation: the n-th allocation a context or batch set-up asks
for is reported as out of memory without being attempted, so nothing reaches
the GPU).  For several positions of the failure:

* pfe_context_setup returns PFE_ENOMEM with the CUDA message, the context is
  left not set up (a build on it is refused with PFE_EINVAL), and the same
  context set up again builds J and K equal to those of a context that never
  failed;
* pfe_batch_setup (two molecules) returns PFE_ENOMEM, the batch refuses builds
  until a set-up succeeds, and its rebuilt batch equals the undisturbed one.
"""
import ctypes

import numpy as np
import pytest
import torch

from polymer_b200 import capi, fock, geometry, scf, system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def waters():
    return [system.build_system(geometry.water_deck(k, seed=70 + k), fock.onee) for k in (2, 3)]


def _pc(sysm):
    return torch.tensor(scf.guess_density(sysm)[0], dtype=torch.float64, device='cuda')


def _build(L, h, sysm, pc):
    """J, K of context h from the contracted density pc through the C ABI."""
    n = sysm.basis.ncgs
    pcf = pc.t().contiguous()
    oc = torch.empty((n, n), dtype=torch.float64, device='cuda')
    ox = torch.empty_like(oc)
    s = torch.cuda.current_stream().cuda_stream
    rc = L.pfe_context_fock_pc(h, ctypes.c_void_p(pcf.data_ptr()), ctypes.c_void_p(oc.data_ptr()),
                               ctypes.c_void_p(ox.data_ptr()), ctypes.c_void_p(s))
    torch.cuda.synchronize()
    return rc, oc, ox


def _close(a, b, rel=1e-12):
    assert float((a - b).abs().max()) <= rel * max(float(b.abs().max()), 1e-300)


@pytest.mark.parametrize('after', [0, 2, 7, 15])
def test_context_setup_recovers_from_allocation_failure(waters, after):
    L = capi.lib()
    sysm = waters[0]
    pc = _pc(sysm)
    ref = fock.DeviceFock(sysm)
    c_ref, x_ref = ref.from_pc(pc)
    ref.close()
    h = ctypes.c_void_p()
    capi.check(L, L.pfe_context_create(0, ctypes.byref(h)))
    try:
        a, keep = sysm.pfe_args(None, None)
        L.pfe_debug_fail_allocation(after)
        rc = L.pfe_context_setup(h, ctypes.byref(a))
        L.pfe_debug_fail_allocation(-1)
        assert rc == -5, (rc, capi.last_error(L))
        assert 'out of memory' in capi.last_error(L)
        rc, _, _ = _build(L, h, sysm, pc)
        assert rc == -1 and 'not set up' in capi.last_error(L)
        capi.check(L, L.pfe_context_setup(h, ctypes.byref(a)))
        rc, oc, ox = _build(L, h, sysm, pc)
        assert rc == 0, capi.last_error(L)
        _close(oc.t(), c_ref)
        _close(ox.t(), x_ref)
    finally:
        L.pfe_debug_fail_allocation(-1)
        L.pfe_context_destroy(h)


@pytest.mark.parametrize('after', [1, 12])
def test_batch_setup_recovers_from_allocation_failure(waters, after):
    L = capi.lib()
    ref = fock.DeviceBatch(waters, 0)
    pc = torch.zeros_like(ref.p_c)
    for k, s in enumerate(waters):
        ref.view(pc, k).copy_(_pc(s))
    ref.run_packed(pc, ref.out_c, ref.out_x)
    torch.cuda.synchronize()
    c_ref, x_ref = ref.out_c.clone(), ref.out_x.clone()
    off = list(ref.off)
    ref.close()
    h = ctypes.c_void_p()
    capi.check(L, L.pfe_batch_create(0, ctypes.byref(h)))
    try:
        args, keep = [], []
        for s in waters:
            a, kp = s.pfe_args(None, None)
            args.append(a)
            keep.append(kp)
        arr = (capi.PfeArgs * len(args))(*args)
        L.pfe_debug_fail_allocation(after)
        rc = L.pfe_batch_setup(h, arr, len(args))
        L.pfe_debug_fail_allocation(-1)
        assert rc == -5, (rc, capi.last_error(L))
        assert 'out of memory' in capi.last_error(L)
        outc, outx = torch.empty_like(pc), torch.empty_like(pc)
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = L.pfe_batch_fock_pc(h, ctypes.c_void_p(pc.data_ptr()), ctypes.c_void_p(outc.data_ptr()),
                                 ctypes.c_void_p(outx.data_ptr()), s)
        assert rc == -1
        capi.check(L, L.pfe_batch_setup(h, arr, len(args)))
        o = (ctypes.c_int64 * (len(args) + 1))()
        assert L.pfe_batch_offsets(h, o) == len(args) and list(o) == off
        capi.check(L, L.pfe_batch_fock_pc(h, ctypes.c_void_p(pc.data_ptr()), ctypes.c_void_p(outc.data_ptr()),
                                          ctypes.c_void_p(outx.data_ptr()), s))
        torch.cuda.synchronize()
        _close(outc, c_ref)
        _close(outx, x_ref)
    finally:
        L.pfe_debug_fail_allocation(-1)
        L.pfe_batch_destroy(h)


GRADIENT = '''
import ctypes, sys
import numpy as np
from polymer_b200 import capi, fock, geometry, system
L = capi.lib()
s, other = [system.build_system(geometry.water_deck(1, seed=k), fock.onee) for k in (80, 81)]
def density(t):
    return (t.basis.cc.T @ np.eye(t.basis.ncgs) @ t.basis.cc)[None]
def gradient():
    return np.concatenate(fock.fourindex_eri_gradient(s, density(s)))
j0, k0 = fock.fourindex_eri(s, density(s))          # the set-up of this geometry
L.pfe_debug_fail_allocation(int(sys.argv[1]))
try:
    gradient()
    raise SystemExit('the failure was not reported')
except capi.FockError as e:
    assert e.code == -5, e
L.pfe_debug_fail_allocation(-1)
j1, k1 = fock.fourindex_eri(s, density(s))
g1 = gradient()
fock.fourindex_eri(other, density(other))           # another geometry, then this one set up again
g2 = gradient()
for a, b in ((j1, j0), (k1, k0), (g1, g2)):
    assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
'''


@pytest.mark.parametrize('after', [0, 1, 2, 12, 40])
def test_gradient_recovers_from_allocation_failure(after):
    """The gradient's scratch (0, 1) and the upload of one of its tables (2 and up: in a process of its own,
    since tables are uploaded once) fail: nothing has been launched, the status is PFE_ENOMEM, and later builds
    and gradients on the same context are those of an undisturbed one."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, '-c', GRADIENT, str(after)], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize('tile, together', [(0, 0), (16 << 20, 1)])
def test_setup_without_room_for_the_stored_integrals_takes_less(waters, tile, together):
    """The failure moved through every allocation of a set-up: PFE_ENOMEM, but at the memory of the stored
    integrals, of which a set-up then takes less (instead of a buffer per class one for all, whose build has the
    same launches; instead of tiles of 16 MiB ones of 4, whose build has more) and builds the same."""
    L = capi.lib()
    sysm = waters[1]
    pc = _pc(sysm)
    ref = fock.DeviceFock(sysm)
    c_ref, x_ref = ref.from_pc(pc)
    ref.close()
    absorbed = []   # (position, launches) of the set-ups that succeeded
    L.pfe_debug_integral_memory(tile, together)
    try:
        for after in range(1000):
            h = ctypes.c_void_p()
            capi.check(L, L.pfe_context_create(0, ctypes.byref(h)))
            a, keep = sysm.pfe_args(None, None)
            L.pfe_debug_fail_allocation(after)
            rc = L.pfe_context_setup(h, ctypes.byref(a))
            L.pfe_debug_fail_allocation(-1)
            if rc == 0:
                c = capi.PfeCensus()
                capi.check(L, L.pfe_context_census(h, ctypes.byref(c)))
                rc, oc, ox = _build(L, h, sysm, pc)
                assert rc == 0, capi.last_error(L)
                _close(oc.t(), c_ref)
                _close(ox.t(), x_ref)
                absorbed.append((after, c.kernel_launches))
            else:
                assert rc == -5, (after, rc, capi.last_error(L))
            L.pfe_context_destroy(h)
            if len(absorbed) == 2:   # the second lies beyond the set-up's last allocation
                break
    finally:
        L.pfe_debug_fail_allocation(-1)
        L.pfe_debug_integral_memory(0, 0)
    (first, less), (last, whole) = absorbed
    assert last == first + 2   # one allocation, that of the chunk flags, comes after the integrals'
    assert less > whole if tile else less == whole
