"""C = alpha op(A) op(B) + beta C for any alpha and beta (cblas_dgemm's contract),
on both sides of the product's shape rules: outputs of few 8 x 8 tiles with a
long inner dimension, single tiles, several 64 x 64 tiles with ragged edges.

Tolerance, element by element: k + 4 roundings of the terms' magnitudes,
(k + 4) u (|alpha| |A| |B| + |beta| |C|) with u = 2^-52."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(5, 7, 3), (8, 8, 100), (13, 9, 200), (64, 64, 64), (70, 50, 33), (130, 67, 5)]
ALPHA = [0.0, 1.0, -1.0, -2.0, 1e-200]
BETA = [0.0, 1.0, -3.0, 1e200]


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_gemm_any_alpha_beta(gpu_lib, m, n, k, ta, tb):
    import torch
    rng = np.random.default_rng(m + 2 * n + 3 * k)
    A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()       # column-major
    dA, dB = dev(A.T if ta else A), dev(B.T if tb else B)
    p = lambda t: C.c_void_p(t.data_ptr())
    for alpha in ALPHA:
        for beta in BETA:
            dC = dev(C0)
            rc = gpu_lib.frank_gemm_batched(m, n, k, 1, alpha, p(dA), k if ta else m, 0, ta, p(dB), n if tb else k, 0,
                                            tb, beta, p(dC), m, 0, None)
            assert rc == 0, gpu_lib.frank_last_error()
            bound = (k + 4) * 2.0 ** -52 * (abs(alpha) * (np.abs(A) @ np.abs(B)) + abs(beta) * np.abs(C0))
            err = np.abs(dC.cpu().numpy().T - (alpha * (A @ B) + beta * C0))
            assert np.all(err <= bound), (alpha, beta)


def test_gemm_beta_zero_does_not_read_c(gpu_lib):
    """beta = 0 overwrites C, whatever it holds; so does alpha = 0 with beta = 0."""
    import torch
    p = lambda t: C.c_void_p(t.data_ptr())
    for m, k in ((8, 100), (70, 33)):
        a = torch.ones((k, m), dtype=torch.float64, device="cuda")
        for alpha in (1.0, 0.0, -2.0):
            c = torch.full((m, m), float("nan"), dtype=torch.float64, device="cuda")
            assert gpu_lib.frank_gemm_batched(m, m, k, 1, alpha, p(a), m, 0, 0, p(a), m, 0, 1, 0.0, p(c), m, 0,
                                              None) == 0
            assert torch.equal(c, torch.full_like(c, alpha * k))
