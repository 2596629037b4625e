"""Device memory: what the large FP64 products and the gauge moves take."""
import ctypes as ct
import threading

import pytest

from gpu_util import device_pointers, device_rand, heff_dev

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module")
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    return nutcracker_b200


def _in_thread(f):
    """f in a thread of its own, which has its own context and arenas."""
    out = {}

    def run():
        out["value"] = f()

    t = threading.Thread(target=run)
    t.start()
    t.join()
    return out["value"]


def test_product_without_room_for_residues(lib):
    """A chi = 448 product (64 MB of workspace) with 170 MB of the device free (22 for the test):
    the integers' 166 MB cannot be had, the FP64 product can."""
    import torch
    from nutcracker_b200 import operators

    op, b = operators.heisenberg(4)[1], 448
    args = (op, device_rand((op.cl, b, b), 1), device_rand((op.cr, b, b), 2), device_rand((op.d, b, b), 3))
    ref = heff_dev(lib, *args)
    graded = (op, args[1], args[2], args[3] * torch.logspace(0, -12, b, dtype=torch.float64, device="cuda")[None, :, None])
    heff_dev(lib, graded[0], graded[1], graded[2], graded[3].contiguous())   # every kernel is loaded
    _in_thread(lambda: lib.lib.nc_synchronize())
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 170 * MB, dtype=torch.uint8, device="cuda")
    try:
        y = _in_thread(lambda: heff_dev(lib, *args))
    finally:
        del hog
        torch.cuda.empty_cache()
    assert float((y - ref).norm() / ref.norm()) < 1e-13


def test_a_second_qr_shape_keeps_its_own_buffers_only(lib):
    """What one more 2048 x 1024 plan adds: its matrix, Q and the reflectors
    (33.5 MB each), R and the compact-WY factor (16.8 MB each) and 12 MB of
    panel scratch, in arena blocks of 64 and 128 MB; the integers of Q's
    products (270 MB) belong to the thread, not to the shape."""
    import torch

    A, B = device_rand((2, 1024, 1024), 1), device_rand((2, 1024, 1024), 2)
    oA, oB = torch.empty_like(A), torch.empty_like(B)
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (1024, 1024, 1024, 2, 2)]

    def moves():
        free = []
        for direction in (1, -1):
            for _ in range(2):
                assert lib.lib.nc_gauge_move_dev(ct.c_int(direction), *dims, *device_pointers(A, B, oA, oB)) == 0
            assert lib.lib.nc_synchronize() == 0
            free.append(torch.cuda.mem_get_info()[0])
        return free[0] - free[1]

    assert _in_thread(moves) <= 224 * MB


def test_footprint_covers_a_chain(lib):
    """Admission's estimate against what a thread of its own takes for a chain
    through two sweeps (every gauge move's plan among it)."""
    import torch
    from nutcracker_b200 import operators
    from nutcracker_b200.chain import Chain
    from nutcracker_b200.serve import footprint_bytes

    ops = operators.heisenberg(22)

    def run():
        lib.lib.nc_synchronize()
        before = torch.cuda.mem_get_info()[0]
        chain = Chain(ops, initial_bandwidth_dimension=512, seed=1)
        chain.perform_optimization_sweep()
        chain.perform_optimization_sweep()
        return before - torch.cuda.mem_get_info()[0]

    torch.cuda.empty_cache()
    used = _in_thread(run)
    print("used", used / MB, "estimate", footprint_bytes(ops, initial_bandwidth_dimension=512) / MB)
    assert used <= footprint_bytes(ops, initial_bandwidth_dimension=512)
