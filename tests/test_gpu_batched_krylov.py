"""Batched Lanczos over its projected problem's sizes: the smallest basis, odd
and even ones (the Jacobi pairing pads odd sizes) and the largest.

Reference: exact diagonalisation.  The sweeps run in FP64 to the default
1e-12 relative energy change at bond dimensions that represent the chains
exactly, so the energy's error is a few sweeps' change, below 1e-9 per site.
"""
import numpy as np
import pytest

from oracle import ed, mpo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", [4, 7, 16, 23, 24])
def test_krylov_dimension(krylov):
    from nutcracker_b200.batched import Batch

    rng = np.random.default_rng(31)
    chains = [(n, mpo.xxz_random(n, rng)) for n in (6, 7)]
    with Batch([ops for _, ops in chains], [2 ** (n // 2) for n, _ in chains], seeds=[1, 2], precision=0,
               krylov_dimension=krylov, maximum_sweeps=60) as b:
        res = b.solve()
    for (n, ops), r in zip(chains, res):
        w, _ = ed.lowest_levels(ops, 1)
        assert abs(r["energy"] - w[0]) / n <= 1e-9
