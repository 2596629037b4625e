"""Gauge moves over several 64-column blocks: shapes at the edges of the blocks,
of the eight-column sub-blocks and of the cluster's 128-row slices, tall and
square, both directions, and rank-deficient and zero columns.

Checked against LAPACK's Householder QR (same sign convention) where the site
has full rank: rounding differences of either grow with its condition number
(about 10 for these random sites), so 1e-11 is asked.  For rank-deficient
sites Q is not unique; the normalised site is orthonormal and the pair's
product unchanged, to 1e-12.
"""
import ctypes as ct

import numpy as np
import pytest

from test_gpu_residue import _rand, _rel, lib  # noqa: F811,F401

pytestmark = pytest.mark.gpu


def _move(lib, direction, A, B):  # noqa: F811
    import torch

    dl, bl, bm = A.shape
    dr, _, br = B.shape
    oA, oB = torch.empty_like(A), torch.empty_like(B)
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (bl, bm, br, dl, dr)]
    assert lib.lib.nc_gauge_move_dev(ct.c_int(direction), *dims,
                                     *[ct.c_void_p(t.data_ptr()) for t in (A, B, oA, oB)]) == 0
    assert lib.lib.nc_synchronize() == 0
    return oA, oB


@pytest.mark.parametrize("bl,bm,br,d", [(33, 65, 40, 2), (72, 72, 70, 2), (100, 127, 90, 2), (64, 128, 64, 2),
                                        (129, 129, 128, 2), (200, 193, 150, 3), (256, 256, 256, 2), (420, 300, 64, 3),
                                        (520, 515, 500, 2), (1024, 1000, 200, 2)])
def test_against_lapack(lib, bl, bm, br, d):  # noqa: F811
    import torch

    A, B = _rand((d, bl, bm), 1), _rand((d, bm, br), 2)
    oA, oB = _move(lib, 1, A, B)
    q, r = np.linalg.qr(A.reshape(d * bl, bm).conj().cpu().numpy())
    assert _rel(oA, torch.from_numpy(q.conj().reshape(d, bl, bm)).cuda()) < 1e-11
    assert _rel(oB, torch.einsum("smr,km->skr", B, torch.from_numpy(r).cuda().conj())) < 1e-11
    # the mirror image: right-normalise a site of the same matrix
    B2 = A.transpose(1, 2).contiguous()          # (d, bm, bl): site (bl, bm, d)
    A2 = B.transpose(1, 2).contiguous()          # (d, br, bm)
    oA2, oB2 = _move(lib, -1, A2, B2)
    assert _rel(oB2, torch.from_numpy(q.conj().reshape(d, bl, bm)).cuda().transpose(1, 2)) < 1e-11
    assert _rel(oA2, torch.einsum("slm,km->slk", A2, torch.from_numpy(r).cuda().conj())) < 1e-11


@pytest.mark.parametrize("kind", ["zero_columns", "low_rank", "real"])
@pytest.mark.parametrize("b", [80, 200])
def test_rank_deficient(lib, b, kind):  # noqa: F811
    import torch

    A, B = _rand((2, b, b), 5), _rand((2, b, b), 6)
    if kind == "zero_columns":
        A[:, :, 3:40] = 0
        A[:, :, 66] = 0
    elif kind == "low_rank":
        A = torch.einsum("alr,rm->alm", A[:, :, :20], A[0, :20, :]).contiguous()
    else:
        A = A.real.to(A.dtype)
    oA, oB = _move(lib, 1, A, B)
    eye = torch.eye(b, dtype=A.dtype, device="cuda")
    assert _rel(torch.einsum("alm,aln->mn", oA, oA.conj()), eye) < 1e-12
    assert _rel(torch.einsum("alm,bmr->albr", oA, oB), torch.einsum("alm,bmr->albr", A, B)) < 1e-12
