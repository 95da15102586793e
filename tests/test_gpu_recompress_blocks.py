"""Recompression at block orders and ranks at the edges of its layouts.

Split targets (one CTA per side of the bases) equal targets on one CTA bit for bit
also for block orders that no vector load divides, where a side lies in shared
memory in one and in scratch in the other."""
import numpy as np
import pytest

import oracle.frank_oracle as fo

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
