"""Thick restarts of the largest sites: the new basis is a product of millions of
rows and a handful of columns, at and above the row count where the smallest
GEMM tile no longer fits a launch grid (16 x 65535 rows).

H = diag over the left index with 9 distinct values, so the lowest eigenvalue is
known; six basis vectors do not hold the Krylov space, the solve has to restart.
The solver stops at a residual of 1e-12 |theta|; the eigenvalue of a Hermitian
matrix is then within 3e-12, 1e-10 is asked.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bl,br,d", [(1020, 1028, 1), (1024, 1024, 2)])
def test_restart_of_a_large_site(bl, br, d):
    import nutcracker_b200 as nb

    rng = np.random.default_rng(9)
    L = np.zeros((bl, bl, 1), complex, order="F")
    L[:, :, 0] = np.diag(np.linspace(-3.0, 5.0, 9)[np.arange(bl) % 9])
    R = np.zeros((br, br, 1), complex, order="F")
    R[:, :, 0] = np.eye(br)
    W = np.asfortranarray(np.eye(d)[:, :, None].astype(complex))
    idx = np.ones((2, 1), np.uint32, order="F")
    guess = rng.normal(size=(br, bl, d)) + 0j
    nb.set_krylov_dimension(6)
    try:
        info, its, ev, x, normal = nb.Core.optimize(bl, br, 1, 1, d, L, 1, idx, W, R, 0, 0, bl * br * d, None, None,
                                                    None, "SR", 1e-12, 1000, guess / np.linalg.norm(guess))
    finally:
        nb.set_krylov_dimension(24)
    assert info == 0 and its > 6
    assert abs(ev + 3.0) < 1e-10 and abs(normal - 1) < 1e-12
    assert np.linalg.norm(x[:, np.arange(bl) % 9 != 0, :]) < 1e-5
