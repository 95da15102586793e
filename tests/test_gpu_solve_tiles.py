"""The solves and the H-matvec at the edges of their tiles: blocks that take
the direct path and the ring, odd block sizes (no 16-byte copies) and ones that
are multiples of the boxes, ragged last blocks, ranks around 16 columns and 56
inner indexes, dense off-diagonal blocks, one to nine right-hand sides (nine
take two passes), FP64 and mixed plans; and the largest blocks.

Tolerances: a product of n terms rounds to n * 2.2e-16 of |A| |x| (entrywise);
the matrices are diagonally dominant with a condition number below 10, their
factors are truncated at 1e-13 (FP64) or 1e-5 (mixed, FP32), so solves agree to
1e-10 and 1e-3."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.2e-16


def _matrix(n, nb, rank, admis, seed, **kw):
    from frank_b200 import BLRMatrix
    rng = np.random.default_rng(seed)
    M = BLRMatrix(n, nb, admis=admis, **kw)
    for i in range(nb):
        for j in range(nb):
            bi, bj = M.block_size(i), M.block_size(j)
            if M.is_lowrank(i, j):
                U, _ = np.linalg.qr(rng.standard_normal((bi, rank)))
                V, _ = np.linalg.qr(rng.standard_normal((bj, rank)))
                M.set_lowrank(i, j, U, rng.standard_normal((rank, rank)) / (2 * nb * rank), V.T)
            else:
                a = rng.standard_normal((bi, bj)) / (4 * nb * np.sqrt(max(bi, bj)))
                M.set_dense(i, j, a + (2.0 * np.eye(bi) if i == j else 0.0))
    return M


def _device(M, f, B):
    import torch
    d = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    f(d)
    torch.cuda.synchronize()
    return d.cpu().numpy().T


CASES = [   # n, nb, max_rank, rank, nrhs, admis
    (97, 3, 33, 1, 1, 0.0), (97, 3, 33, 17, 3, 0.0), (128, 4, 32, 16, 8, 1.0), (515, 2, 16, 15, 9, 0.0),
    (300, 2, 150, 57, 2, 0.0), (768, 3, 256, 56, 8, 0.0), (771, 3, 0, 41, 5, 1.0), (1026, 2, 513, 16, 4, 0.0),
    (1024, 2, 512, 130, 9, 1.0), (1500, 2, 750, 33, 8, 0.0),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,nb,kmax,rank,nrhs,admis", CASES)
def test_solve_and_matvec(gpu_lib, n, nb, kmax, rank, nrhs, admis, precision):
    import torch
    eps, tol = (1e-13, 1e-10) if precision == "fp64" else (1e-5, 1e-3)
    M = _matrix(n, nb, rank, admis, n + rank, eps=eps, max_rank=kmax, precision=precision)
    A = M.to_dense()
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, nrhs))
    out = torch.zeros((nrhs, n), dtype=torch.float64, device="cuda")
    _device(M, lambda d: M.matvec_device(d.data_ptr(), out.data_ptr(), nrhs), X)
    assert (np.abs(out.cpu().numpy().T - A @ X) <= n * EPS * (np.abs(A) @ np.abs(X)) + EPS).all()
    M.getrf()
    for At, solve in ((A, M.solve_device), (A.T, M.solve_transpose_device)):
        got = _device(M, lambda d: solve(d.data_ptr(), nrhs), X)
        want = np.linalg.solve(At, X)
        assert (np.linalg.norm(got - want, axis=0) <= tol * np.linalg.norm(want, axis=0)).all()
    # transposed products, through the residual of the transposed refinement (at most 8 right-hand sides)
    X, nrhs = X[:, :8], min(nrhs, 8)
    b, x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda(), torch.zeros((nrhs, n), dtype=torch.float64, device="cuda")
    it, res = C.c_int(), C.c_double()
    assert gpu_lib.frank_blr_refine_transpose_device(M._h, C.c_void_p(b.data_ptr()), n, C.c_void_p(x.data_ptr()), n,
                                                     nrhs, 1e-11, 20, C.byref(it), C.byref(res), None) == 0
    want = np.linalg.solve(A.T, X)
    assert np.linalg.norm(x.cpu().numpy().T - want) <= 1e-9 * np.linalg.norm(want)
    M.close()


def test_the_largest_blocks(gpu_lib):
    n, nrhs = 1619, 9                       # blocks of 810 and 809, the largest accepted
    M = _matrix(n, 2, 20, 0.0, 5, eps=1e-13, max_rank=0)
    A = M.to_dense()
    X = np.random.default_rng(1).standard_normal((n, nrhs))
    got = M.matvec(X)
    assert (np.abs(got - A @ X) <= n * EPS * (np.abs(A) @ np.abs(X)) + EPS).all()
    M.close()
