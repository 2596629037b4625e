"""Site solves long enough to run a Lanczos step beside the previous step's
projected problem: basis sizes around the first such step and the restarts,
every eigenvalue request, sites that end by exhausting a small space, and one
whose space splits (an invariant subspace found on the way).

Reference: dense eigh of the oracle's H_eff.  The solver stops at a residual of
1e-12 |theta|, so its eigenvalue is within 1e-10 of the dense one, relatively.
"""
import numpy as np
import pytest

from oracle import core
from test_gpu_optimize import herm_env, herm_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", [6, 7, 8, 24])
@pytest.mark.parametrize("which", ["SR", "LR", "LM"])
@pytest.mark.parametrize("bl,br,d", [(2, 2, 3), (7, 6, 2), (12, 11, 2)])
def test_against_dense(krylov, which, bl, br, d):
    import nutcracker_b200 as nb

    rng = np.random.default_rng(bl * 100 + br)
    L, R = herm_env(rng, bl, 3), herm_env(rng, br, 3)
    idx, W = herm_mpo(rng, 3, 3, d, 6)
    w = np.linalg.eigvalsh(core.compute_optimization_matrix(bl, br, 3, 3, d, L, idx, W, R))
    want = {"SR": w[0], "LR": w[-1], "LM": w[-1] if abs(w[-1]) > abs(w[0]) else w[0]}[which]
    guess = rng.normal(size=(br, bl, d)) + 1j * rng.normal(size=(br, bl, d))
    nb.set_krylov_dimension(krylov)
    try:
        info, its, ev, x, normal = nb.Core.optimize(bl, br, 3, 3, d, L, 6, idx, W, R, 0, 0, bl * br * d, None, None,
                                                    None, which, 1e-12, 4000, guess / np.linalg.norm(guess))
    finally:
        nb.set_krylov_dimension(24)
    assert info == 0 and its >= min(6, bl * br * d)
    assert abs(ev - want) <= 1e-10 * abs(want) and abs(normal - 1) < 1e-12


def test_invariant_subspace_on_the_way():
    """H = diag over the left index with 9 distinct values: from any guess the
    Krylov space ends after 9 vectors, and the solve has to go on from a random
    one or stop at the right value."""
    import nutcracker_b200 as nb

    bl, br, d = 9, 5, 2
    L = np.zeros((bl, bl, 1), complex, order="F")
    L[:, :, 0] = np.diag(np.linspace(-3.0, 5.0, bl))
    R = np.zeros((br, br, 1), complex, order="F")
    R[:, :, 0] = np.eye(br)
    W = np.asfortranarray(np.eye(d)[:, :, None].astype(complex))
    idx = np.ones((2, 1), np.uint32, order="F")
    rng = np.random.default_rng(3)
    guess = rng.normal(size=(br, bl, d)) + 0j
    info, its, ev, x, _ = nb.Core.optimize(bl, br, 1, 1, d, L, 1, idx, W, R, 0, 0, bl * br * d, None, None, None, "SR",
                                           1e-13, 1000, guess / np.linalg.norm(guess))
    assert info == 0 and abs(ev + 3.0) < 1e-11
    assert np.linalg.norm(x[:, 1:, :]) < 1e-9
