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
