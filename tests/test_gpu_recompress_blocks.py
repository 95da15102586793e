"""Recompression at block orders and ranks at the edges of its layouts.

Split targets (one CTA per side of the bases) equal targets on one CTA bit for bit
also for block orders that no vector load divides, where a side lies in shared
memory in one and in scratch in the other.

Blocks of 513 to 810 rows (panels eight columns wide, four rows a thread) with a
ragged last block, at least three block rows, each core method, projected and
stacked bases, joint ranks whose cores are in shared memory, above it, and above 512
rows: diagonally dominant matrices with condition numbers below 10.  Tolerance: the
factors are truncated at 1e-13 and sum a few hundred terms, so A - L U stays below
1e-11 of A and solves agree to 1e-10; fixed-rank plans hold the exact sums."""
import numpy as np
import pytest

import oracle.frank_oracle as fo
from tests.test_gpu_blr import _factor_error
from tests.test_gpu_solve_tiles import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("b,short,eps", [(333, 5, 1e-5), (401, 2, 1e-5), (501, 0, 1e-4), (272, 1, 1e-6)])
def test_split_targets_match_one_cta_at_any_order(gpu_lib, b, short, eps, precision):
    from frank_b200 import BLRMatrix
    n, nb = 13 * b - short, 13       # plans of fewer block rows do not split targets
    x, _ = fo.morton_sort(np.random.default_rng(b).random((3, n)), 12)
    mats = []
    for grid in (0, 64):
        M = BLRMatrix(n, nb, eps=eps, precision=precision)
        M.build_kernel("laplace", x, eps)
        if grid:
            M.set_grid(grid)         # every target on one CTA
        M.getrf()
        mats.append(M)
    ranks = [M.rank(i, j, 0) for i in range(nb) for j in range(nb) if i != j]
    split = M.tuning()["split_rank"]
    assert sum(split < r <= 23000 // (b + 20) for r in ranks) > 10      # in shared memory on a CTA of its own only
    A, B = mats
    for i in range(nb):
        for j in range(nb):
            ba, bb = A.block(i, j, 1), B.block(i, j, 1)
            if isinstance(ba, tuple):
                assert A.rank(i, j, 1) == B.rank(i, j, 1), (i, j)
                for u, v in zip(ba, bb):
                    assert np.array_equal(u, v), (i, j)
            else:
                assert np.array_equal(ba, bb), (i, j)
    A.close()
    B.close()


CASES = [   # block order, rows missing from the last block, rank of the blocks, algorithm
    (513, 7, 20, "rounded_addition_rrqr_proj"), (513, 0, 90, "rounded_addition_rrqr"), (600, 100, 70, "rounded_addition"),
    (600, 3, 130, "rounded_addition_rrqr_proj"), (600, 1, 270, "rounded_addition_rrqr"), (810, 2, 33, "rounded_addition"),
    (810, 0, 290, "rounded_addition_rrqr_proj"), (810, 5, 75, "rounded_addition_rrqr"), (777, 9, 150, "rounded_addition"),
]


@pytest.mark.parametrize("b,short,rank,alg", CASES)
def test_large_blocks(gpu_lib, b, short, rank, alg):
    n, nb = 3 * b - short, 3
    M = _matrix(n, nb, rank, 0.0, b + rank, eps=1e-13)
    M.set_lra(alg)
    A = M.to_dense()
    M.getrf()
    assert _factor_error(A, M) <= 1e-11
    X = np.random.default_rng(n).standard_normal((n, 2))
    got, want = M.solve(X), np.linalg.solve(A, X)
    assert (np.linalg.norm(got - want, axis=0) <= 1e-10 * np.linalg.norm(want, axis=0)).all()
    x, _, res = M.refine(X, tol=1e-14, maxit=10)
    assert np.linalg.norm(x - want) <= 1e-12 * np.linalg.norm(want)
    M.close()


@pytest.mark.parametrize("b,short,rank", [(513, 7, 8), (640, 0, 45), (810, 1, 100)])
def test_large_blocks_fixed_rank(gpu_lib, b, short, rank):
    """Blocks of rank `rank` in a plan of twice that rank: every sum is exact."""
    n, nb = 3 * b - short, 3
    M = _matrix(n, nb, rank, 0.0, b + rank, eps=0.0, fixed_rank=2 * rank)
    A = M.to_dense()
    M.getrf()
    assert _factor_error(A, M) <= 1e-11
    X = np.random.default_rng(n).standard_normal((n, 2))
    got, want = M.solve(X), np.linalg.solve(A, X)
    assert (np.linalg.norm(got - want, axis=0) <= 1e-10 * np.linalg.norm(want, axis=0)).all()
    M.close()
