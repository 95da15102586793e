"""Construction of H-matrices whose leaves are smaller than the sample of the
larger blocks (leaf < rank + 5 <= 2 leaf): every block within 1e-9 (relative,
Frobenius) of the oracle's LowRank(Dense, rank), as in the other construction
tests."""
import numpy as np
import pytest

import oracle.frank_oracle as fo
from tests.test_gpu_hodlr import _blocks, _points, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,rank", [(64, 8, 8), (128, 8, 5), (256, 16, 16), (1024, 8, 8), (80, 20, 20)])
def test_construction_with_small_leaves(gpu_lib, n, leaf, rank):
    from frank_b200 import HMatrix
    pts = _points(n)
    M = HMatrix(n, leaf, rank)
    M.build_kernel("laplace", pts)
    for key, blk in _blocks(fo.build_hierarchical(fo.laplacend, pts, n, leaf, 2, rank=rank)).items():
        if key[0] == "D":
            np.testing.assert_allclose(M.get_dense(key[1]), blk, rtol=1e-13)
        else:
            U, S, V = M.get_lowrank(key[1], key[2])
            assert _rel(U @ S @ V, blk.dense()) < 1e-9, key
    M.close()
