"""frank_hodlr_stats counts the launches of one factorization (its header's
promise): solves, products and refinements do not add to it, and a second
factorization has the same count."""
import numpy as np
import pytest

import oracle.frank_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,rank,nrhs", [(256, 32, 4, 1), (1024, 64, 16, 33)])
def test_launch_count_is_the_factorizations(gpu_lib, n, leaf, rank, nrhs):
    from frank_b200 import HMatrix
    M = HMatrix(n, leaf, rank)
    M.build_kernel("laplace", np.array([fo.get_sorted_random_vector(n)]))
    x = np.random.default_rng(0).standard_normal((n, nrhs))
    M.matvec(x)
    M.getrf()
    want = M.stats()["launches"]
    assert want > 0
    M.solve(x)
    M.matvec(x)
    M.refine(x, tol=1e-10)
    assert M.stats()["launches"] == want
    M.getrf()
    assert M.stats()["launches"] == want
    M.close()
