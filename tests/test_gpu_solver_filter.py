"""Site solves with as many projectors as the filter's two forms meet at: up to
eight vectors go through one launch, more through two.  Sites of one block of
elements and of several.

Reference: dense eigh of the oracle's H_eff on the space orthogonal to the
projectors.  The solver stops at a residual of 1e-12 |theta|, so its eigenvalue
is within 1e-10 of the dense one, relatively; the filter leaves an overlap with
the projectors of a few roundings, below 1e-12.
"""
import numpy as np
import pytest

from oracle import core
from test_gpu_optimize import dense_ref, herm_env, herm_mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nproj", [7, 8, 9, 16])
@pytest.mark.parametrize("bl,br,d", [(6, 5, 2), (15, 13, 2)])
def test_projector_counts(nproj, bl, br, d):
    import nutcracker_b200 as nb

    rng = np.random.default_rng(nproj * 100 + bl)
    n = bl * br * d
    L, R = herm_env(rng, bl, 3), herm_env(rng, br, 3)
    idx, W = herm_mpo(rng, 3, 3, d, 6)
    vecs = np.asfortranarray(rng.normal(size=(n, nproj)) + 1j * rng.normal(size=(n, nproj)))
    refl, rank, tau, swaps = core.convert_vectors_to_reflectors(n, nproj, vecs)
    proj = (nproj, nproj, n - rank, refl, tau, swaps)
    want = dense_ref(bl, br, 3, 3, d, L, idx, W, R, "SR", proj)[0]
    y = rng.normal(size=n - rank) + 1j * rng.normal(size=n - rank)
    guess = core.unproject_from_orthogonal_space(n, nproj, nproj, n - rank, refl, tau, swaps, y / np.linalg.norm(y))
    guess = np.asfortranarray(np.reshape(guess, (br, bl, d), order="F"))
    info, _, ev, x, normal = nb.Core.optimize(bl, br, 3, 3, d, L, 6, idx, W, R, nproj, nproj, n - rank, refl, tau,
                                              swaps, "SR", 1e-12, 4000, guess)
    assert info == 0 and rank == nproj
    assert abs(ev - want) <= 1e-10 * abs(want) and abs(normal - 1) < 1e-12
    assert core.compute_overlap_with_projectors(nproj, nproj, refl, tau, swaps, n, x) < 1e-12
