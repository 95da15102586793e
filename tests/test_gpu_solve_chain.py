"""The solves' chain of launches, each of which may begin before the end of the one
before it: blocks on both sides of the line between the direct form and the ring
(64 rows), ranks around the transposed core's boxes (56 rows, 64 columns), steps
whose targets are all dense (every CTA of the inner launch has nothing to do), one
block, and solves that follow each other without a wait, on one stream and on two.

Tolerance as in the other solve tests: diagonally dominant matrices with condition
numbers below 10, factors truncated at 1e-13, so solves agree to 1e-10."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_solve_tiles import _matrix

pytestmark = pytest.mark.gpu

CASES = [   # n, nb, max_rank, rank, nrhs, admis
    (64 * 4, 4, 64, 30, 3, 0.0), (65 * 4 - 9, 4, 65, 30, 3, 0.0), (130 * 3, 3, 130, 55, 1, 0.0),
    (130 * 3 - 1, 3, 130, 57, 8, 0.0), (260 * 3, 3, 260, 64, 2, 0.0), (260 * 3, 3, 260, 65, 5, 0.0),
    (300 * 3, 3, 300, 120, 4, 0.0), (90 * 5, 5, 90, 4, 2, 10.0), (40 * 6, 6, 40, 4, 2, 10.0), (150, 1, 0, 0, 3, 0.0),
]


@pytest.mark.parametrize("n,nb,kmax,rank,nrhs,admis", CASES)
def test_solve_chain(gpu_lib, n, nb, kmax, rank, nrhs, admis):
    import torch
    M = _matrix(n, nb, rank, admis, n + rank, eps=1e-13, max_rank=kmax)
    A = M.to_dense()
    M.getrf()
    X = np.random.default_rng(n).standard_normal((n, nrhs))
    x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    for At, solve in ((A, M.solve_device), (A.T, M.solve_transpose_device)):
        # three solves one after another in the same buffer: A^-3 x
        y = x.clone()
        for _ in range(3):
            solve(y.data_ptr(), nrhs)
        torch.cuda.synchronize()
        want = np.linalg.solve(At, np.linalg.solve(At, np.linalg.solve(At, X)))
        got = y.cpu().numpy().T
        assert (np.linalg.norm(got - want, axis=0) <= 3e-10 * np.linalg.norm(want, axis=0)).all()
    M.close()


def test_solves_on_two_streams(gpu_lib):
    """Two plans solving at once give what each gives by itself, bit for bit."""
    import torch
    plans = [_matrix(600, 4, 20, 0.0, 1, eps=1e-13, max_rank=150), _matrix(48 * 8, 8, 6, 0.0, 2, eps=1e-13, max_rank=48)]
    rhs = []
    for M in plans:
        M.getrf()
        rhs.append(torch.from_numpy(np.random.default_rng(M.n).standard_normal((4, M.n))).cuda())

    def run(streams):
        out = [r.clone() for r in rhs]
        torch.cuda.synchronize()
        for _ in range(20):
            for M, o, s in zip(plans, out, streams):
                M.solve_device(o.data_ptr(), 4, stream=s)
                M.solve_transpose_device(o.data_ptr(), 4, stream=s)
        torch.cuda.synchronize()
        return out

    alone = run([None, None])
    side = [torch.cuda.Stream() for _ in plans]
    both = run([C.c_void_p(s.cuda_stream) for s in side])
    for a, b in zip(alone, both):
        assert torch.equal(a, b)
    for M in plans:
        M.close()
