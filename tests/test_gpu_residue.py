"""FP64 products through residues on the int8 tensor cores (large H_eff products
and environment updates) against plain complex128 torch products.

Sizes: from just above the smallest product that takes this route, at edges of
the 128 x 256 output tile, the 128-byte K stage and the 16 x 128 conversion
tile, and remainders of all of them.

Tolerance: operands are rounded to 2^-59 of their row's (column's) 2-norm per
component, so an output is within 4 sqrt(K) 2^-59 |a_m| |b_n| of exact; torch's
own FP64 sums add about sqrt(K) 2^-53 of the same scale.  Relative to the
2-norm of a whole random result (about |a| |b|) both are below 1e-14 for the K
used here (at most 3200); 1e-13 is asked.
"""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    return nutcracker_b200


def _rand(shape, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)


def _ptrs(*t):
    return [ct.c_void_p(x.data_ptr()) for x in t]


def _heff(lib, op, L, R, psi):
    import torch

    d, bl, br = psi.shape
    W = torch.from_numpy(op.W.ravel(order="F").copy()).cuda()
    idx = torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda()
    y = torch.empty_like(psi)
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (bl, br, op.cl, op.cr, d, op.nnz)]
    assert lib.lib.nc_heff_apply_dev(*dims, *_ptrs(idx, W, L, R, psi, y)) == 0
    assert lib.lib.nc_synchronize() == 0
    return y


def _heff_ref(op, L, R, psi):
    import torch

    W = torch.from_numpy(np.ascontiguousarray(op.W)).cuda()
    T = torch.einsum("ali,kjl->kaji", psi, L)
    out = torch.zeros_like(psi)
    for n in range(op.nnz):
        f, t = int(op.idx[0, n]) - 1, int(op.idx[1, n]) - 1
        out += torch.einsum("bjr,rx->bjx", torch.einsum("ab,ajr->bjr", W[:, :, n], T[f]), R[t])
    return out


def _rel(x, y):
    return float((x - y).norm() / y.norm())


@pytest.mark.parametrize("model,bl,br", [("heisenberg", 256, 256), ("heisenberg", 257, 255), ("heisenberg", 384, 300),
                                         ("ising", 512, 389), ("spin1", 243, 301), ("heisenberg", 640, 513)])
def test_heff_and_environments(lib, model, bl, br):
    import torch
    from nutcracker_b200 import operators

    op = {"heisenberg": operators.heisenberg, "ising": lambda n: operators.ferromagnetic_transverse_ising(n, 1.2),
          "spin1": operators.heisenberg_spin1}[model](4)[1]
    L, R = _rand((op.cl, bl, bl), 1), _rand((op.cr, br, br), 2)
    psi = _rand((op.d, bl, br), 3)
    assert _rel(_heff(lib, op, L, R, psi), _heff_ref(op, L, R, psi)) < 1e-13
    W = torch.from_numpy(op.W.ravel(order="F").copy()).cuda()
    idx = torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda()
    Wm = torch.from_numpy(np.ascontiguousarray(op.W)).cuda()
    dims = [ct.c_uint32(v) for v in (bl, br, op.cl, op.cr, op.d, op.nnz)]
    for side, env, b, c in ((0, L, br, op.cr), (1, R, bl, op.cl)):
        out = torch.empty((c, b, b), dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        assert lib.lib.nc_env_update_dev(ct.c_int(side), ct.c_int(0), *dims, *_ptrs(idx, W, env, psi, out)) == 0
        assert lib.lib.nc_synchronize() == 0
        ref = torch.zeros_like(out)
        for n in range(op.nnz):
            f, t = int(op.idx[0, n]) - 1, int(op.idx[1, n]) - 1
            if side == 0:
                U = torch.einsum("ab,aji->bji", Wm[:, :, n], torch.einsum("ali,jl->aji", psi, L[f]))
                ref[t] += torch.einsum("bjr,bjx->xr", U, psi.conj())
            else:
                Z = torch.einsum("ab,bxr->axr", Wm[:, :, n], torch.einsum("bxq,rq->bxr", psi.conj(), R[t]))
                ref[f] += torch.einsum("axr,ayr->yx", Z, psi)
        assert _rel(out, ref) < 1e-13


def test_scales_zeros_and_non_finite(lib):
    """Rows far apart in scale keep their own relative accuracy; zero rows give
    zeros; a NaN or infinity stays in the outputs that it reaches."""
    import torch
    from nutcracker_b200.operators import construct_operator_site

    op = construct_operator_site(1, 1, 1, [(1, 1, np.eye(1))])
    n = 520
    G, L, R = _rand((1, n, n), 4), _rand((1, n, n), 5), _rand((1, n, n), 6)
    # y[j, x] = sum R[r, x] psi[l, r] L[j, l]: scales on j and x leave every sum's terms alike
    s = torch.tensor([10.0 ** (150 * np.sin(i)) for i in range(n)], dtype=torch.float64, device="cuda")
    ref = _heff_ref(op, L, R, G)
    y = _heff(lib, op, (L * s[None, :, None]).contiguous(), (R / s[None, None, :]).contiguous(), G)
    got = y / s[None, :, None] * s[None, None, :]
    assert float(((got - ref).abs().amax() / ref.abs().amax())) < 1e-13
    L0 = L.clone()
    L0[0, 7, :] = 0
    y = _heff(lib, op, L0, R, G)
    assert torch.count_nonzero(y[0, 7]) == 0 and _rel(y, _heff_ref(op, L0, R, G)) < 1e-13
    for bad in (float("nan"), float("inf")):
        L0 = L.clone()
        L0[0, 11, 3] = bad
        y = _heff(lib, op, L0, R, G)
        assert not torch.isfinite(torch.view_as_real(y[0, 11])).any()
        keep = [j for j in range(n) if j != 11]
        assert torch.isfinite(torch.view_as_real(y[0, keep])).all() and _rel(y[0, keep], ref[0, keep]) < 1e-13
