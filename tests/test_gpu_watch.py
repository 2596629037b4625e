"""Expired device waits: bounded, reported once, to the thread whose work it was.

A test switch makes a kernel withhold one arrival, so that a wait runs out after
a short limit (2 ms) and the kernel returns.  No fault is involved.
"""
import ctypes as ct
import threading

import pytest

from gpu_util import device_rand, heff_dev

pytestmark = pytest.mark.gpu
TIMEOUT = 1004
RESIDUE = 2


@pytest.fixture()
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    yield nutcracker_b200
    assert nutcracker_b200.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    nutcracker_b200.lib.nc_synchronize()


def _mute(lib, kinds):
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000), ct.c_uint32(kinds)) == 0


def _product():
    """Operands of an H_eff product that runs through residues."""
    from nutcracker_b200 import operators

    op = operators.heisenberg(4)[1]
    b = 448
    return op, device_rand((op.cl, b, b), 1), device_rand((op.cr, b, b), 2), device_rand((op.d, b, b), 3)


def test_other_threads_do_not_take_it(lib):
    """Another thread's synchronisation neither fails for this thread's expired
    wait nor hides it."""
    import torch

    args = _product()
    ref = heff_dev(lib, *args)
    _mute(lib, RESIDUE)
    status, _ = heff_dev(lib, *args, wait=False)
    assert status == 0
    torch.cuda.synchronize()
    seen = {}

    def other():
        seen["before"] = lib.lib.nc_synchronize()
        seen["y"] = heff_dev(lib, *args)
        seen["after"] = lib.lib.nc_synchronize()

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert seen["before"] == 0 and seen["after"] == 0 and torch.equal(seen["y"], ref)
    assert lib.lib.nc_synchronize() == TIMEOUT and b"residue GEMM" in lib.lib.nc_last_error()
    assert lib.lib.nc_synchronize() == 0


def test_residue_gemm_recovers(lib):
    import torch

    args = _product()
    ref = heff_dev(lib, *args)
    _mute(lib, RESIDUE)
    for _ in range(2):
        status, _ = heff_dev(lib, *args, wait=False)
        assert status == 0
    assert lib.lib.nc_synchronize() == TIMEOUT
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    assert torch.equal(heff_dev(lib, *args), ref)
