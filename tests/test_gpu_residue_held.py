"""Products through residues keep FP64 operands: what the integers do not hold
goes to the FP64 product.

With identity environments an H_eff product returns psi, and every FP64
operation on the way is exact, so whatever differs was lost in the operands.  A
component above 2^-24 of its row's (or column's) norm is held; below, it may be
rounded by 2^-77 of the norm, once in each of the two products, and each
product's result is rounded to FP64 (relative 2^-53).  Operands with more than
one rounded component in 2^15, and non-finite ones, must come out exact.
"""
import ctypes as ct

import numpy as np
import pytest

from gpu_util import device_pointers, device_rand, heff_dev

pytestmark = pytest.mark.gpu
N = 944   # 944^3 complex multiplications are just enough for the route


@pytest.fixture(scope="module")
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    return nutcracker_b200


def _identity_product(lib, psi):
    import torch
    from nutcracker_b200.operators import construct_operator_site

    op = construct_operator_site(1, 1, 1, [(1, 1, np.eye(1))])
    eye = torch.eye(N, dtype=torch.complex128, device="cuda")[None].contiguous()
    return heff_dev(lib, op, eye, eye, psi.contiguous())


def _check(y, psi):
    """Every component within the bounds above."""
    import torch

    row = psi.abs().square().sum(1, keepdim=True).sqrt()   # over the left bond, then over the right one
    col = psi.abs().square().sum(2, keepdim=True).sqrt()
    bound = 2.0 ** -52 * psi.abs() + 2.0 ** -77 * np.sqrt(2) * (row + col)
    assert bool(((y - psi).abs() <= bound).all())
    assert torch.isfinite(torch.view_as_real(y)).all()


@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("least", [1.0, 1e-2, 1e-4, 1e-8, 1e-12, 1e-16])
def test_graded_bond(lib, least, axis):
    """Weights 1 .. least on a contracted bond."""
    import torch

    w = torch.logspace(0, np.log10(least), N, dtype=torch.float64, device="cuda")
    psi = device_rand((1, N, N), 1) * (w[None, :, None] if axis == 1 else w[None, None, :])
    y = _identity_product(lib, psi)
    _check(y, psi)
    last = (y - psi).abs() / psi.abs()
    last = last[0, -1] if axis == 1 else last[0, :, -1]
    assert float(last.median()) <= 2.0 ** -52


def test_one_graded_column(lib):
    """The first product is refused; the second has that column as a row of its own."""
    psi = device_rand((1, N, N), 2)
    psi[0, 77] *= 1e-12
    y = _identity_product(lib, psi)
    _check(y, psi)
    bound = 2.0 ** -53 * psi[0, 77].abs() + 2.0 ** -76 * psi[0, 77].norm()
    assert bool(((y[0, 77] - psi[0, 77]).abs() <= bound).all())


def test_small_rows(lib):
    """Rows whose scale leaves the exponent range of a power of two."""
    psi = device_rand((1, N, N), 3)
    psi[0, :, 7] *= 2.0 ** -990
    psi[0, 9, :] *= 2.0 ** -1000
    assert bool((_identity_product(lib, psi) == psi).all())


def test_ordinary_operands_take_residues(lib):
    """One small component among random ones: rounded, so not the FP64 product's
    result, and by no more than the bound."""
    psi = device_rand((1, N, N), 4)
    psi[0, 5, 6] = (1 / 3 + 1j / 7) * 2.0 ** -40
    y = _identity_product(lib, psi)
    _check(y, psi)
    assert complex(y[0, 5, 6]) != complex(psi[0, 5, 6])


def test_long_sums_near_the_moduli(lib):
    """16000 terms (the longest sum through residues), almost all residues p - 1."""
    import torch
    from nutcracker_b200.operators import construct_operator_site

    br, bl, cr = 1000, 128, 16
    op = construct_operator_site(1, 1, cr, [(1, k + 1, np.eye(1)) for k in range(cr)])
    L = torch.eye(bl, dtype=torch.complex128, device="cuda")[None].contiguous()
    psi = torch.full((1, bl, br), -1 - 1j, dtype=torch.complex128, device="cuda")
    R = torch.full((cr, br, br), -1 - 1j, dtype=torch.complex128, device="cuda")
    psi[0, :, 0] = 2.0 ** 74      # norms just above 2^76: a unit stays a unit
    R[0, 0, :] = 2.0 ** 76
    y = torch.view_as_real(heff_dev(lib, op, L, R, psi))
    # 2^150 - 15 * 2^74 (1 + i) + 2 i * 999 * 16
    assert float((y[..., 0] - 2.0 ** 150).abs().max()) <= 2.0 ** 98
    assert float((y[..., 1] - (2 * 999 * 16 - 15 * 2.0 ** 74)).abs().max()) <= 2.0 ** 41


@pytest.mark.parametrize("side", [0, 1])
def test_graded_environment_update(lib, side):
    """An environment update of a graded site by an identity environment is the
    site's Gram matrix; FP64 sums keep each entry to the sizes of its own terms."""
    import torch
    from nutcracker_b200.operators import construct_operator_site

    op = construct_operator_site(2, 1, 1, [(1, 1, np.eye(2))])
    w = torch.logspace(0, -10, N, dtype=torch.float64, device="cuda")
    psi = device_rand((2, N, N), 5) * (w[None, None, :] if side == 0 else w[None, :, None])
    env = torch.eye(N, dtype=torch.complex128, device="cuda")[None].contiguous()
    out = torch.empty_like(env)
    W = torch.from_numpy(op.W.ravel(order="F").copy()).cuda()
    idx = torch.from_numpy(op.idx.ravel(order="F").astype(np.int32)).cuda()
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (N, N, 1, 1, 2, op.nnz)]
    assert lib.lib.nc_env_update_dev(ct.c_int(side), ct.c_int(0), *dims, *device_pointers(idx, W, env, psi, out)) == 0
    assert lib.lib.nc_synchronize() == 0
    x = psi.transpose(1, 2) if side == 0 else psi
    ref = torch.einsum("axj,ayj->yx", x, x.conj()) if side == 0 else torch.einsum("axj,ayj->yx", x.conj(), x)
    size = torch.einsum("axj,ayj->yx", x.abs(), x.abs())
    assert bool(((out[0] - ref).abs() <= 2 * N * 2.0 ** -53 * 4 * size).all())


def test_norms_out_of_range_of_squares(lib):
    """Rows whose squares overflow or vanish keep their own accuracy."""
    psi = device_rand((1, N, N), 6)
    psi[0, :, 3] *= 2.0 ** 600
    psi[0, :, 4] *= 2.0 ** -600
    y = _identity_product(lib, psi)
    _check(y[:, :, [4]] * 2.0 ** 600, psi[:, :, [4]] * 2.0 ** 600)
    _check(y[:, :, [3]] * 2.0 ** -600, psi[:, :, [3]] * 2.0 ** -600)


@pytest.mark.parametrize("model,bl,br", [("heisenberg", 448, 448), ("heisenberg", 449, 447), ("heisenberg", 513, 640),
                                         ("heisenberg", 641, 385), ("ising", 700, 512), ("spin1", 385, 449)])
def test_shapes(lib, model, bl, br):
    """Edges of the 128 x 256 output tile, the 128-byte K stage and the 16 x 128
    conversion tile, against plain complex128 products.  Operands of random
    elements are held, so an output is one rounding from exact; the reference's
    own sums of K <= 3200 terms stay below sqrt(K) 2^-53 of the result's norm,
    6e-15: 1e-13 is asked."""
    import torch
    from nutcracker_b200 import operators

    op = {"heisenberg": operators.heisenberg, "ising": lambda n: operators.ferromagnetic_transverse_ising(n, 1.2),
          "spin1": operators.heisenberg_spin1}[model](4)[1]
    W = torch.from_numpy(np.ascontiguousarray(op.W)).cuda()
    L, R, psi = device_rand((op.cl, bl, bl), 1), device_rand((op.cr, br, br), 2), device_rand((op.d, bl, br), 3)
    T = torch.einsum("ali,kjl->kaji", psi, L)
    ref = torch.zeros_like(psi)
    for n in range(op.nnz):
        f, t = int(op.idx[0, n]) - 1, int(op.idx[1, n]) - 1
        ref += torch.einsum("bjr,rx->bjx", torch.einsum("ab,ajr->bjr", W[:, :, n], T[f]), R[t])
    y = heff_dev(lib, op, L, R, psi)
    assert float((y - ref).norm() / ref.norm()) < 1e-13
