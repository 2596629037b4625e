"""The sparse-MPO mixes over operator and site shapes: few and many channels
(more than a staged tile holds), every physical dimension, duplicate matrices
between the same indices, positions around the tiles' edges.

FP64 against plain complex128 torch, 1e-12 (sums of at most a few hundred
terms, rounding below 1e-14).  Precision form against the same reference: its
products keep 22 bits and accumulate in FP32, about 1e-6 of the result's
2-norm at these sizes; 1e-5 is asked.
"""
import ctypes as ct

import numpy as np
import pytest

from gpu_util import random_mpo_site
from test_gpu_residue import _heff, _heff_ref, _rand, _rel, lib  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cl,cr,d,nnz,bl,br", [(1, 1, 1, 1, 5, 3), (3, 7, 4, 20, 17, 33), (40, 3, 3, 64, 9, 20),
                                               (2, 130, 3, 60, 12, 7), (130, 2, 4, 64, 6, 11), (5, 5, 2, 12, 130, 129)])
def test_mixes(lib, cl, cr, d, nnz, bl, br):  # noqa: F811
    import torch
    from nutcracker_b200.operators import OperatorSite

    idx, Wn = random_mpo_site(np.random.default_rng(nnz), cl, cr, d, nnz)
    op = OperatorSite(d, cl, cr, idx, Wn)
    L, R, psi = _rand((cl, bl, bl), 1), _rand((cr, br, br), 2), _rand((d, bl, br), 3)
    ref = _heff_ref(op, L, R, psi)
    assert _rel(_heff(lib, op, L, R, psi), ref) < 1e-12
    W = torch.from_numpy(op.W.ravel(order="F").copy()).cuda()
    di = torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda()
    Wm = torch.from_numpy(np.ascontiguousarray(op.W)).cuda()
    dims = [ct.c_uint32(v) for v in (bl, br, cl, cr, d, nnz)]
    ptr = [ct.c_void_p(t.data_ptr()) for t in (di, W, L, R, psi)]
    y = torch.empty_like(psi)
    torch.cuda.synchronize()
    assert lib.lib.nc_heff_apply_mixed_dev(*dims, *ptr, ct.c_void_p(y.data_ptr())) == 0
    assert _rel(y, ref) < 1e-5
    for side, env, b, c in ((0, L, br, cr), (1, R, bl, cl)):
        want = torch.zeros((c, b, b), dtype=L.dtype, device="cuda")
        for n in range(nnz):
            f, t = int(op.idx[0, n]) - 1, int(op.idx[1, n]) - 1
            if side == 0:
                U = torch.einsum("ab,aji->bji", Wm[:, :, n], torch.einsum("ali,jl->aji", psi, L[f]))
                want[t] += torch.einsum("bjr,bjx->xr", U, psi.conj())
            else:
                Z = torch.einsum("ab,bxr->axr", Wm[:, :, n], torch.einsum("bxq,rq->bxr", psi.conj(), R[t]))
                want[f] += torch.einsum("axr,ayr->yx", Z, psi)
        for mixed, tol in ((0, 1e-12), (1, 1e-5)):
            out = torch.empty_like(want)
            torch.cuda.synchronize()
            args = ptr[:2] + [ct.c_void_p(env.data_ptr()), ptr[4], ct.c_void_p(out.data_ptr())]
            assert lib.lib.nc_env_update_dev(ct.c_int(side), ct.c_int(mixed), *dims, *args) == 0
            assert lib.lib.nc_synchronize() == 0
            assert _rel(out, want) < tol
