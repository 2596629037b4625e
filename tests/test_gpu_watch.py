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
QR = 4


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


@pytest.mark.parametrize("bl,bm", [(60, 96), (130, 125), (520, 515)])
def test_qr_panel_recovers(lib, bl, bm):
    """One to nine CTAs a panel; the first call runs the panels directly, the
    second from the recorded graph, with the waits running out in both."""
    import torch
    from gpu_util import device_pointers

    A, B = device_rand((2, bl, bm), 1), device_rand((2, bm, 70), 2)
    dims = [ct.c_uint32(v) for v in (bl, bm, 70, 2, 2)]

    def move():
        oA, oB = torch.empty_like(A), torch.empty_like(B)
        torch.cuda.synchronize()
        status = lib.lib.nc_gauge_move_dev(ct.c_int(1), *dims, *device_pointers(A, B, oA, oB))
        return status, oA, oB

    for _ in range(2):
        _mute(lib, QR)
        assert move()[0] == 0
        assert lib.lib.nc_synchronize() == TIMEOUT and b"cluster QR" in lib.lib.nc_last_error()
        assert lib.lib.nc_synchronize() == 0
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    status, oA, oB = move()
    assert status == 0 and lib.lib.nc_synchronize() == 0
    eye = torch.eye(bm, dtype=A.dtype, device="cuda")
    assert float((torch.einsum("alm,aln->mn", oA, oA.conj()) - eye).norm() / eye.norm()) < 1e-12
    ref = torch.einsum("alm,bmr->albr", A, B)
    assert float((torch.einsum("alm,bmr->albr", oA, oB) - ref).norm() / ref.norm()) < 1e-12


def test_host_buffer_call_reports(lib):
    """A call on host buffers waits for its own work: it reports, and the next one is right."""
    import numpy as np

    rng = np.random.default_rng(3)
    A = np.asfortranarray(rng.normal(size=(100, 90, 2)) + 1j * rng.normal(size=(100, 90, 2)))   # (bm, bl, d)
    B = np.asfortranarray(rng.normal(size=(60, 100, 2)) + 1j * rng.normal(size=(60, 100, 2)))
    args = (90, 100, 60, 2, 2, A, B)
    good = lib.Core.norm_denorm_going_right(*args)
    _mute(lib, QR)
    with pytest.raises(lib.NutcrackerError, match="cluster QR"):
        lib.Core.norm_denorm_going_right(*args)
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    again = lib.Core.norm_denorm_going_right(*args)
    assert all(np.array_equal(x, y) for x, y in zip(good[-2:], again[-2:]))


def test_chain_calls_report(lib):
    """A chain's calls that hand out or keep the state answer for the moves that
    made it; a growth that went wrong leaves the chain as it was."""
    import numpy as np
    from nutcracker_b200 import operators
    from nutcracker_b200.chain import Chain

    chain = Chain(operators.heisenberg(14), initial_bandwidth_dimension=80, seed=3)
    chain.perform_optimization_sweep()
    energy = chain.get_energy()
    site = chain.get_site(0)
    _mute(lib, QR)
    with pytest.raises(lib.NutcrackerError, match="cluster QR"):
        chain.increase_bandwidth_dimension(100)
    with pytest.raises(lib.NutcrackerError, match="cluster QR"):
        chain.construct_and_add_projector_from_state()
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    info = chain.info()
    assert info["bandwidth_dimension"] == 80 and info["number_of_projectors"] == 0
    assert np.array_equal(chain.get_site(0), site)
    assert abs(chain.compute_expectation_value() - energy) < 1e-9 * abs(energy)
    chain.increase_bandwidth_dimension(100)
    assert abs(chain.compute_expectation_value() - energy) < 1e-9 * abs(energy)
    _mute(lib, QR)
    chain.move_to(7)
    assert lib.lib.nc_test_device_wait(ct.c_uint64(2_000_000_000), ct.c_uint32(0)) == 0
    with pytest.raises(lib.NutcrackerError, match="cluster QR"):
        chain.get_site(7)


def test_two_threads_at_once(lib):
    """Products through residues and panels of both threads in flight together:
    the bits of a thread alone."""
    import torch
    from gpu_util import device_pointers

    args = _product()
    A, B = device_rand((2, 300, 290), 4), device_rand((2, 290, 200), 5)
    dims = [ct.c_uint32(v) for v in (300, 290, 200, 2, 2)]

    def work():
        out = []
        for _ in range(4):
            y = heff_dev(lib, *args)
            oA, oB = torch.empty_like(A), torch.empty_like(B)
            torch.cuda.current_stream().synchronize()
            assert lib.lib.nc_gauge_move_dev(ct.c_int(1), *dims, *device_pointers(A, B, oA, oB)) == 0
            assert lib.lib.nc_synchronize() == 0
            out.append((y, oA, oB))
        return out

    ref = work()[0]
    results = [None, None]

    def run(i):
        results[i] = work()

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out in results:
        assert out is not None
        for got in out:
            assert all(torch.equal(x, y) for x, y in zip(got, ref))
