"""Helpers shared by the GPU parity tests."""
import numpy as np


def rand_c(rng, shape):
    return np.asfortranarray(rng.normal(size=shape) + 1j * rng.normal(size=shape))


def rel_err(got, want):
    got = np.asarray(got).ravel(order="F")
    want = np.asarray(want).ravel(order="F")
    den = max(np.linalg.norm(want), 1e-300)
    return float(np.linalg.norm(got - want) / den)


def random_mpo_site(rng, cl, cr, d, nnz):
    idx = np.asfortranarray(np.stack([rng.integers(1, cl + 1, nnz), rng.integers(1, cr + 1, nnz)]).astype(np.uint32))
    W = rand_c(rng, (d, d, nnz))
    return idx, W


def device_rand(shape, seed):
    """Random complex128 tensor on the GPU."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)


def device_pointers(*tensors):
    import ctypes as ct

    return [ct.c_void_p(t.data_ptr()) for t in tensors]


def heff_dev(lib, op, L, R, psi, wait=True):
    """H_eff psi through nc_heff_apply_dev; L (cl,bl,bl), R (cr,br,br), psi (d,bl,br)."""
    import ctypes as ct

    import torch

    d, bl, br = psi.shape
    W = torch.from_numpy(np.ascontiguousarray(op.W.ravel(order="F"))).cuda()
    idx = torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda()
    y = torch.empty_like(psi)
    torch.cuda.current_stream().synchronize()   # of this thread's work only: others may be recording graphs
    dims = [ct.c_uint32(v) for v in (bl, br, op.cl, op.cr, d, op.nnz)]
    status = lib.lib.nc_heff_apply_dev(*dims, *device_pointers(idx, W, L, R, psi, y))
    if not wait:
        return status, y
    assert status == 0 and lib.lib.nc_synchronize() == 0
    return y
