"""Batched Lanczos on vectors of several chunks (2048 elements each): whole
chunks and a ragged last one, with a basis so short that every solve restarts.

Reference: exact diagonalisation where the bond dimension represents the chain
exactly; a smaller bond dimension can only lie above it.  The sweeps run in
FP64 to the default 1e-12 relative energy change, so the energy's error is a
few sweeps' change, below 1e-9 per site.  A chain gives the same energy alone
and beside others, to the last bit.
"""
import numpy as np
import pytest

from oracle import ed, mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", [5, 20])
def test_several_chunks(krylov):
    from nutcracker_b200.batched import Batch

    rng = np.random.default_rng(41)
    n = 13
    ops = mpo.xxz_random(n, rng)
    small = mpo.xxz_random(6, rng)
    members = [(ops, 64, 1), (ops, 47, 2), (small, 8, 3)]   # site vectors of up to 8192, 4418 and 128 elements

    def energies(members):
        with Batch([m[0] for m in members], [m[1] for m in members], seeds=[m[2] for m in members], precision=0,
                   krylov_dimension=krylov, maximum_sweeps=60) as b:
            return [r["energy"] for r in b.solve()]

    together = energies(members)
    w, _ = ed.lowest_levels(ops, 1)
    assert abs(together[0] - w[0]) / n <= 1e-9
    assert together[1] >= w[0] - 1e-9 * n
    w, _ = ed.lowest_levels(small, 1)
    assert abs(together[2] - w[0]) / 6 <= 1e-9
    assert energies(members[1:2])[0] == together[1]
