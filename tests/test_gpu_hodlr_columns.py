"""H-matrix products and solves of many columns: the buffers stay bounded (the
columns go in passes), and each column is what it is by itself.

Bound: n = 1024 in leaves of 8 has 128 leaves; partial products and T2 of one pass
of 128 columns take 128 blocks x 8 x 128 x 8 bytes = 1 MB each, so 8 MB with the
allocator's granularity; 4000 columns at once would take 65 MB.  Columns: the
operations of a column do not depend on the others, so only the order of a sum of
n products may differ, 1e-13 relative with room to spare."""
import ctypes as C

import numpy as np
import pytest

import oracle.frank_oracle as fo

pytestmark = pytest.mark.gpu


def test_many_columns_in_bounded_memory(gpu_lib):
    import torch
    from frank_b200 import HMatrix
    n, leaf, rank, nrhs = 1024, 8, 8, 4000
    M = HMatrix(n, leaf, rank)
    M.build_kernel("laplace", np.array([fo.get_sorted_random_vector(n)]))
    M.getrf()
    x = torch.randn((nrhs, n), dtype=torch.float64, device="cuda")
    y, z = torch.empty_like(x), x.clone()
    p = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    assert gpu_lib.frank_hodlr_matvec_device(M._h, p(x), n, p(y), n, nrhs, None) == 0, gpu_lib.frank_last_error()
    assert gpu_lib.frank_hodlr_solve_device(M._h, p(z), n, nrhs, None) == 0, gpu_lib.frank_last_error()
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
    for c in (0, 7, 8, 31, 32, 127, 128, 129, 255, 256, 3967, 3999):
        y1, z1 = torch.empty_like(x[0]), x[c].clone()
        assert gpu_lib.frank_hodlr_matvec_device(M._h, p(x[c]), n, p(y1), n, 1, None) == 0
        assert gpu_lib.frank_hodlr_solve_device(M._h, p(z1), n, 1, None) == 0
        assert torch.norm(y[c] - y1) <= 1e-13 * torch.norm(y1)
        assert torch.norm(z[c] - z1) <= 1e-13 * torch.norm(z1)
    M.close()
