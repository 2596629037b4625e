"""Rounding errors of a gauge move's QR over several blocks, in extended precision.

The bounds are the mean errors of a Householder QR whose panels are factorised a
column at a time, with every dot product in short chains (measured on the same
sites, 8 seeds): summing in another order may not cost accuracy.
"""
import ctypes as ct

import numpy as np
import pytest

from gpu_util import device_pointers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import nutcracker_b200
    import torch

    torch.cuda.init()
    nutcracker_b200.lib.nc_use_own_stream()
    return nutcracker_b200


def _qr(lib, X):
    """X (m, n) = Q R through a move right of the site X^H and an identity neighbour."""
    import torch

    m, n = X.shape
    A = X.conj().resolve_conj().reshape(1, m, n).contiguous()
    B = torch.eye(n, dtype=X.dtype, device="cuda").reshape(1, n, n).contiguous()
    oA, oB = torch.empty_like(A), torch.empty_like(B)
    torch.cuda.synchronize()
    dims = [ct.c_uint32(v) for v in (m, n, n, 1, 1)]
    assert lib.lib.nc_gauge_move_dev(ct.c_int(1), *dims, *device_pointers(A, B, oA, oB)) == 0
    assert lib.lib.nc_synchronize() == 0
    return oA[0].conj().resolve_conj(), oB[0].conj().resolve_conj()


@pytest.mark.parametrize("m,n,graded,orthogonality,residual", [
    (260, 125, True, 1.089e-14, 8.20e-16), (260, 125, False, 1.104e-14, 9.49e-16),
    (192, 96, True, 8.05e-15, 7.35e-16), (192, 96, False, 8.17e-15, 8.00e-16),
    (256, 128, True, 1.138e-14, 8.37e-16), (256, 128, False, 1.145e-14, 9.54e-16)])
def test_errors(lib, m, n, graded, orthogonality, residual):
    import torch

    o = r = 0.0
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        X = torch.randn(m, n, dtype=torch.complex128, device="cuda", generator=g)
        if graded:
            X = torch.fft.fft(X * torch.logspace(0, -4, n, dtype=torch.float64, device="cuda"), dim=1, norm="ortho")
        Q, R, A = [t.cpu().numpy().astype(np.clongdouble) for t in (*_qr(lib, X), X)]
        o += np.linalg.norm((Q.conj().T @ Q - np.eye(n)).astype(complex)) / 8
        r += np.linalg.norm((A - Q @ R).astype(complex)) / np.linalg.norm(X.cpu().numpy()) / 8
    assert o <= orthogonality and r <= residual, (o, r)


@pytest.mark.parametrize("kind", ["columns", "rows", "sectors"])
def test_graded_site_at_full_size(lib, kind):
    """A 2048 x 1024 site whose columns or rows span 12 orders, or with blocks
    that vanish to rounding: Q orthonormal, and every column of A its own column
    of QR, however small.  A Householder QR's errors per column are about
    sqrt(m) 2^-53 of the column, 5e-15, and sqrt(n) times that in Q^H Q - I."""
    import torch

    m, n = 2048, 1024
    g = torch.Generator(device="cuda").manual_seed(0)
    X = torch.randn(m, n, dtype=torch.complex128, device="cuda", generator=g)
    if kind == "rows":
        X = X * torch.logspace(0, -12, m, dtype=torch.float64, device="cuda")[:, None]
    else:
        if kind == "sectors":
            rows = torch.randint(0, 9, (m,), device="cuda", generator=g)
            cols = torch.randint(0, 7, (n,), device="cuda", generator=g)
            X = torch.where(rows[:, None] == cols[None, :], X, X * 1e-17)
        X = X * torch.logspace(0, -12, n, dtype=torch.float64, device="cuda")
    Q, R = _qr(lib, X)
    assert float((Q.conj().T @ Q - torch.eye(n, device="cuda")).norm()) <= 1.6e-13
    assert float(((X - Q @ R).norm(dim=0) / X.norm(dim=0)).max()) <= 5e-15
