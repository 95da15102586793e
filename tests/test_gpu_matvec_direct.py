"""The H-matvec on both sides of the rule that picks its form: grids of many small
blocks (128 threads per block), blocks above 128 rows (256 threads), blocks of
whole boxes with up to four right-hand sides (the ring) and more; odd block sizes,
a ragged last block, ranks that are not multiples of a tile, a rank of one, dense
off-diagonal blocks.

Tolerance as for the other products: n terms round to n * 2.2e-16 of |A| |x|
(entrywise), A the matrix that the plan holds."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_solve_tiles import EPS, _matrix

pytestmark = pytest.mark.gpu

CASES = [   # n, nb, rank, nrhs, admis, fixed rank plan
    (24 * 8, 8, 3, 1, 0.0, False), (33 * 32 - 5, 32, 7, 2, 0.0, False), (128 * 6, 6, 20, 9, 1.0, False),
    (129 * 5 - 40, 5, 33, 3, 0.0, False), (160 * 32, 32, 5, 1, 0.0, False), (161 * 4 - 7, 4, 1, 8, 1.0, True),
    (257 * 3, 3, 65, 4, 0.0, False), (512 * 16, 16, 9, 5, 0.0, False), (512 * 16, 16, 9, 1, 0.0, True),
    (809 * 3 - 2, 3, 40, 8, 0.0, False),
]


@pytest.mark.parametrize("n,nb,rank,nrhs,admis,fixed", CASES)
def test_matvec(gpu_lib, n, nb, rank, nrhs, admis, fixed):
    import torch
    kw = dict(fixed_rank=rank, eps=0.0) if fixed else dict(eps=1e-10, max_rank=rank)
    M = _matrix(n, nb, rank, admis, n + nrhs, **kw)
    A = M.to_dense()
    X = np.random.default_rng(n).standard_normal((n, nrhs))
    x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    y = torch.full_like(x, float("nan"))
    p = lambda t: C.c_void_p(t.data_ptr())
    for At, product in ((A, gpu_lib.frank_blr_matvec_device), (A.T, gpu_lib.frank_blr_matvec_transpose_device)):
        assert product(M._h, p(x), n, p(y), n, nrhs, None) == 0, gpu_lib.frank_last_error()
        torch.cuda.synchronize()
        assert (np.abs(y.cpu().numpy().T - At @ X) <= n * EPS * (np.abs(At) @ np.abs(X)) + EPS).all()
    # one column by itself
    assert gpu_lib.frank_blr_matvec_device(M._h, p(x[-1]), n, p(y[0]), n, 1, None) == 0
    torch.cuda.synchronize()
    assert (np.abs(y[0].cpu().numpy() - A @ X[:, -1]) <= n * EPS * (np.abs(A) @ np.abs(X[:, -1])) + EPS).all()
    M.close()
