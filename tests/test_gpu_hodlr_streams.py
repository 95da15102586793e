"""H-matrix calls on a non-blocking stream while the default stream is busy: the
first product and the first solve allocate and zero the chunk counters of the
level kernels, which has to be ordered with the launches that use them.

The kernels sum in a fixed order, so the results equal those of a second
H-matrix of the same blocks used on the idle default stream, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle.frank_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,rank,nrhs", [(2048, 64, 8, 1), (4096, 128, 16, 40)])
def test_first_calls_on_a_side_stream(gpu_lib, n, leaf, rank, nrhs):
    import torch
    from frank_b200 import HMatrix
    pts = np.array([fo.get_sorted_random_vector(n)])
    M, ref = HMatrix(n, leaf, rank), HMatrix(n, leaf, rank)
    for h in (M, ref):
        h.build_kernel("laplace", pts)
    x = torch.from_numpy(np.random.default_rng(n).standard_normal((nrhs, n))).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())

    def product_and_solve(h, stream, busy):
        y, z = torch.empty_like(x), x.clone()
        h.getrf()
        torch.cuda.synchronize()
        busy()
        assert gpu_lib.frank_hodlr_matvec_device(h._h, p(x), n, p(y), n, nrhs, stream) == 0, gpu_lib.frank_last_error()
        busy()
        assert gpu_lib.frank_hodlr_solve_device(h._h, p(z), n, nrhs, stream) == 0, gpu_lib.frank_last_error()
        torch.cuda.synchronize()
        return y, z

    a = torch.randn((4096, 4096), device="cuda")

    def busy():
        b = a
        for _ in range(40):        # some 40 ms of FP32 products on the default stream
            b = torch.mm(a, b)
            b = b / b.abs().max()

    side = torch.cuda.Stream()
    got = product_and_solve(M, C.c_void_p(side.cuda_stream), busy)
    want = product_and_solve(ref, None, lambda: None)
    for g, w in zip(got, want):
        assert torch.equal(g, w)
    M.close()
    ref.close()
