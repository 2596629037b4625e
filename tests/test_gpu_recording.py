"""Gauge moves whose graph cannot be recorded: the move itself is right.

The first move of a shape runs directly and is recorded afterwards; on the
legacy default stream nothing can be recorded, and another thread's device-wide
synchronisation ends a recording in progress.
"""
import ctypes as ct
import threading

import pytest

from gpu_util import device_pointers, device_rand

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    yield nutcracker_b200
    nutcracker_b200.lib.nc_use_own_stream()


def _move(lib, A, B):
    import torch

    (dl, bl, bm), (dr, _, br) = A.shape, B.shape
    oA, oB = torch.zeros_like(A), torch.zeros_like(B)
    torch.cuda.current_stream().synchronize()
    dims = [ct.c_uint32(v) for v in (bl, bm, br, dl, dr)]
    status = lib.lib.nc_gauge_move_dev(ct.c_int(1), *dims, *device_pointers(A, B, oA, oB))
    return status, lib.lib.nc_synchronize(), oA, oB


def _right(A, B, oA, oB):
    import torch

    eye = torch.eye(A.shape[2], dtype=A.dtype, device="cuda")
    pair = torch.einsum("alm,bmr->albr", A, B)
    return (float((torch.einsum("alm,aln->mn", oA, oA.conj()) - eye).norm() / eye.norm()) < 1e-12
            and float((torch.einsum("alm,bmr->albr", oA, oB) - pair).norm() / pair.norm()) < 1e-12)


@pytest.mark.parametrize("bl,bm", [(60, 97), (200, 193)])
def test_legacy_default_stream(lib, bl, bm):
    A, B = device_rand((2, bl, bm), 1), device_rand((2, bm, 70), 2)
    assert lib.lib.nc_set_stream(None) == 0
    for _ in range(2):
        status, sync, oA, oB = _move(lib, A, B)
        assert status == 0 and sync == 0 and _right(A, B, oA, oB)
    assert lib.lib.nc_use_own_stream() == 0
    for _ in range(2):   # the shape can still be recorded, and replayed, elsewhere
        status, sync, oA, oB = _move(lib, A, B)
        assert status == 0 and sync == 0 and _right(A, B, oA, oB)


def test_device_synchronisation_in_another_thread(lib):
    """Sixteen shapes recorded while another thread keeps synchronising the device
    (whose calls CUDA refuses while a recording is in progress)."""
    import torch

    stop = threading.Event()

    def hammer():
        while not stop.is_set():
            try:
                torch.cuda.synchronize()
            except RuntimeError:
                pass

    t = threading.Thread(target=hammer)
    t.start()
    try:
        results = []
        for k in range(16):
            A, B = device_rand((2, 160 + k, 150 + k), k), device_rand((2, 150 + k, 70), 50 + k)
            for _ in range(2):
                results.append((A, B, *_move(lib, A, B)))
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    for A, B, status, sync, oA, oB in results:
        assert status == 0 and sync == 0 and _right(A, B, oA, oB)
