"""The tiled leaf LU and its explicit inverses at the edges of its tiles:
orders around one panel (32 columns), around the register panels' limit (512
rows; larger blocks take 16-column panels of two rows per thread) and the
smallest and largest accepted ones, on random blocks (which pivot) and on a
block whose exchanges all fall into the last panel.

Tolerances: LU of a random block of order n grows at most about n^(2/3), and
each entry carries n rounding errors, so entries agree with dgetrf's to
n^2 * 2.2e-16 * max|LU|; a solve through the explicit inverses agrees with
LAPACK's to n * cond(A) * 2.2e-16, with a factor 10 for the inverses."""
import numpy as np
import pytest
from scipy.linalg import lapack

pytestmark = pytest.mark.gpu
EPS = 2.2e-16


def _factor(A):
    from frank_b200 import BLRMatrix
    M = BLRMatrix(A.shape[0], 1, eps=1e-12)
    M.set_dense(0, 0, A)
    M.getrf()
    return M


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 95, 129, 480, 511, 512, 513, 527, 600, 810])
def test_leaf_edges(gpu_lib, n):
    rng = np.random.default_rng(1000 + n)
    A = rng.standard_normal((n, n))
    M = _factor(A)
    lu, piv, _ = lapack.dgetrf(np.asfortranarray(A))
    assert (M.pivots(0) == piv + 1).all()
    got = M.block(0, 0, which=1)
    np.testing.assert_allclose(got, lu, rtol=0, atol=n * n * EPS * np.abs(lu).max() + EPS)
    b = rng.standard_normal((n, 3))
    want = np.linalg.solve(A, b)
    err = np.linalg.norm(M.solve(b) - want) / np.linalg.norm(want)
    assert err <= 10 * n * EPS * np.linalg.cond(A)
    M.close()


@pytest.mark.parametrize("n", [40, 300, 530])
def test_exchanges_in_the_last_panel_only(gpu_lib, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 4.0 * n * np.eye(n)
    k = n - 4
    A[k:, k:] = rng.standard_normal((4, 4))       # the last columns pivot, the others do not
    A[k:, :k] *= 1e-3
    M = _factor(A)
    lu, piv, _ = lapack.dgetrf(np.asfortranarray(A))
    assert (piv[:k] == np.arange(k)).all() and (piv[k:] != np.arange(k, n)).any()
    assert (M.pivots(0) == piv + 1).all()
    np.testing.assert_allclose(M.block(0, 0, which=1), lu, rtol=0, atol=n * EPS * np.abs(lu).max())
    b = rng.standard_normal((n, 1))
    want = np.linalg.solve(A, b)
    err = np.linalg.norm(M.solve(b) - want) / np.linalg.norm(want)
    assert err <= 10 * n * EPS * np.linalg.cond(A)
    M.close()
