"""The FP64 complex GEMM's tile shapes, through H_eff products and gauge moves
at sizes on and around the tiles' edges (16, 32, 64, 128), against plain
complex128 torch.

Tolerance: sums of at most 5 * 193 terms in FP64 on both sides, rounding error
about sqrt(K) 2^-53 of the result's 2-norm, below 1e-14; 1e-12 is asked.
"""
import pytest

from test_gpu_residue import _heff, _heff_ref, _rand, _rel, lib  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bl,br", [(1, 2), (2, 1), (15, 17), (16, 16), (33, 31), (48, 64), (65, 63), (97, 95),
                                   (128, 129), (150, 97), (161, 160), (193, 177)])
def test_heff(lib, bl, br):  # noqa: F811
    from nutcracker_b200 import operators

    op = operators.heisenberg(4)[1]
    L, R, psi = _rand((op.cl, bl, bl), bl), _rand((op.cr, br, br), br), _rand((op.d, bl, br), 7)
    assert _rel(_heff(lib, op, L, R, psi), _heff_ref(op, L, R, psi)) < 1e-12


@pytest.mark.parametrize("b", [5, 17, 33, 66, 130])
@pytest.mark.parametrize("direction", [1, -1])
def test_gauge_move(lib, direction, b):  # noqa: F811
    import ctypes as ct

    import torch

    A, B = _rand((2, b, b), 3), _rand((2, b, b), 4)          # (br,bl,d) as (d,bl,br)
    oA, oB = torch.empty_like(A), torch.empty_like(B)
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (b, b, b, 2, 2)]
    assert lib.lib.nc_gauge_move_dev(ct.c_int(direction), *dims,
                                     *[ct.c_void_p(t.data_ptr()) for t in (A, B, oA, oB)]) == 0
    assert lib.lib.nc_synchronize() == 0
    two = torch.einsum("alm,bmr->albr", A, B)
    assert _rel(torch.einsum("alm,bmr->albr", oA, oB), two) < 1e-12
    eye = torch.eye(b, dtype=A.dtype, device="cuda")
    q = torch.einsum("alm,aln->mn", oA, oA.conj()) if direction > 0 else torch.einsum("bmr,bnr->mn", oB, oB.conj())
    assert _rel(q, eye) < 1e-12
