"""Inputs that are not finite: the call reports it (as one-sided Jacobi that does
not converge, whose sweeps such values never end) and leaves NaN in the result of
that block, and the other blocks of the batch are what they are without it."""
import ctypes as C

import numpy as np
import pytest

from frank_b200 import _abi

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("alg", ["rounded_addition", "fast_rounded_addition"])
@pytest.mark.parametrize("m,n,k", [(40, 33, 5), (300, 200, 32), (200, 300, 50)])   # joint ranks 10, 64 and 100
@pytest.mark.parametrize("where,value", [("Ua", float("nan")), ("Sb", float("nan")), ("Vb", float("nan")),
                                         ("Sa", float("inf"))])
def test_lowrank_add_not_finite(gpu_lib, alg, m, n, k, where, value):
    import torch
    if value == float("inf") and k > 44:
        pytest.skip("the larger ranks' Jacobi takes an infinite column for converged")
    rng = np.random.default_rng(m)
    count = 3
    rows = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    orth = lambda r: np.stack([np.linalg.qr(rng.standard_normal((r, k)))[0] for _ in range(count)])
    base = dict(Ua=rows(orth(m).swapaxes(1, 2)), Va=rows(orth(n)), Ub=rows(orth(m).swapaxes(1, 2)), Vb=rows(orth(n)),
                Sa=rows(np.stack([np.diag(0.7 ** np.arange(k))] * count)),
                Sb=rows(np.stack([np.diag(0.6 ** np.arange(k))] * count)))

    def add(t):
        t = {key: v.clone() for key, v in t.items()}
        ka = torch.full((count,), k, dtype=torch.int32, device="cuda")
        kb = ka.clone()
        rc = gpu_lib.frank_lowrank_add_batched(
            m, n, count, k, alg.encode(), 0.0, _p(t["Ua"]), m, m * k, _p(t["Sa"]), k, k * k, _p(t["Va"]), k, k * n,
            _p(ka), _p(t["Ub"]), m, m * k, _p(t["Sb"]), k, k * k, _p(t["Vb"]), k, k * n, _p(kb), k, None)
        return rc, [t[key] for key in ("Ua", "Sa", "Va")]

    rc, want = add(base)
    assert rc == 0, gpu_lib.frank_last_error()
    bad = {key: v.clone() for key, v in base.items()}
    bad[where][1, 0, 0] = value
    rc, got = add(bad)
    assert rc == _abi.FRANK_ERR_NOT_CONVERGED
    for g, w in zip(got, want):
        assert torch.equal(g[0], w[0]) and torch.equal(g[2], w[2])
    assert torch.isnan(got[1][1]).any()


@pytest.mark.parametrize("m,n", [(64, 32), (33, 70)])
def test_svd_not_finite(gpu_lib, m, n):
    import torch
    k = min(m, n)
    A = torch.randn((2, n, m), dtype=torch.float64, device="cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")

    def svd(a):
        U, S, V = z(2, k, m), z(2, k), z(2, n, k)
        rc = gpu_lib.frank_svd_batched(m, n, 2, _p(a), m, m * n, _p(U), m, m * k, _p(S), k, _p(V), k, k * n, None)
        return rc, U, S, V

    want = svd(A)
    assert want[0] == 0
    B = A.clone()
    B[1, 3, 2] = float("nan")
    got = svd(B)
    assert got[0] == _abi.FRANK_ERR_NOT_CONVERGED
    for g, w in zip(got[1:], want[1:]):
        assert torch.equal(g[0], w[0])
    assert torch.isnan(got[2][1]).any()
