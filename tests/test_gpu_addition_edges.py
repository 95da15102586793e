"""The LowRank addition and the H-LU's substitutions at the edges of their
tiles: sides of more than one chunk of 512 rows, joint ranks around the largest
that shared memory holds (88), rank-deficient sums; H-matrices with odd leaves,
ranks and right-hand sides above one 32-column tile.

Tolerances: as for the same operations at ordinary sizes (additions 1e-11 of
the operands' norms with equal ranks; H-LU solutions within a factor 10 of the
oracle's error plus 1e-13)."""
import numpy as np
import pytest

import oracle.frank_oracle as fo
from tests.test_gpu_ops import _lr_add

pytestmark = pytest.mark.gpu


def _lowrank(rng, m, n, k, decay):
    U, _ = np.linalg.qr(rng.standard_normal((m, k)))
    V, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return fo.LowRank(U, np.diag(decay ** np.arange(k)), V.T.copy(), k)


@pytest.mark.parametrize("alg", ["rounded_addition", "fast_rounded_addition"])
@pytest.mark.parametrize("m,n,ka,kb", [(511, 513, 8, 8), (512, 1024, 32, 32), (513, 600, 5, 7), (1025, 130, 16, 3),
                                       (1537, 1537, 32, 32), (200, 300, 44, 44), (200, 300, 44, 45), (96, 95, 9, 1)])
def test_lowrank_add_edges(gpu_lib, alg, m, n, ka, kb):
    rng = np.random.default_rng(m + n + ka + kb)
    A, B = _lowrank(rng, m, n, ka, 0.7), _lowrank(rng, m, n, kb, 0.6)
    U, S, V, r = _lr_add(gpu_lib, A, B, alg, 0.0, ka + kb)
    ref = A.copy()
    (fo.fast_rounded_addition if alg == "fast_rounded_addition" else fo.rounded_addition)(ref, B)
    assert r == ref.rank == ka
    np.testing.assert_allclose(U @ S @ V, ref.dense(), rtol=0,
                               atol=1e-11 * (np.linalg.norm(A.dense()) + np.linalg.norm(B.dense())))


@pytest.mark.parametrize("m,n,k", [(64, 48, 6), (700, 520, 20)])
def test_lowrank_add_of_the_same_block(gpu_lib, m, n, k):
    """A + A has the rank of A: half of the joint core is zero."""
    A = _lowrank(np.random.default_rng(k), m, n, k, 0.5)
    for alg in ("rounded_addition", "fast_rounded_addition"):
        U, S, V, r = _lr_add(gpu_lib, A, A.copy(), alg, 0.0, 2 * k)
        assert r == k
        np.testing.assert_allclose(U @ S @ V, 2 * A.dense(), rtol=0, atol=1e-11 * np.linalg.norm(A.dense()))


@pytest.mark.parametrize("leaf,levels,rank,nrhs", [(33, 2, 5, 1), (45, 3, 8, 33), (96, 1, 33, 3), (100, 2, 40, 40),
                                                   (32, 1, 4, 65)])
def test_hlu_edges(gpu_lib, leaf, levels, rank, nrhs):
    from frank_b200 import HMatrix
    n = leaf << levels
    pts = np.array([fo.get_sorted_random_vector(n)])
    M = HMatrix(n, leaf, rank)
    M.build_kernel("laplace", pts)
    H = fo.build_hierarchical(fo.laplacend, pts, n, leaf, 2, rank=rank)
    X = np.random.default_rng(n).standard_normal((n, nrhs))
    B = M.matvec(X)
    ref = np.stack([np.ravel(fo.matvec(H, X[:, c].copy())) for c in range(nrhs)], axis=1)
    assert np.linalg.norm(B - ref) <= 1e-12 * np.linalg.norm(ref)
    M.getrf()
    sol = M.solve(B)
    L, U = fo.getrf(fo.deep_copy(H))
    want = np.stack([np.ravel(fo.solve(L, U, ref[:, c].copy())) for c in range(nrhs)], axis=1)
    for c in range(nrhs):
        assert fo.l2_error(X[:, c], sol[:, c]) <= 10 * fo.l2_error(X[:, c], want[:, c]) + 1e-13
    M.close()
