"""Batches of more small blocks than SMs, which take the variants with several CTAs
an SM: LowRank additions (both algorithms, fixed rank and accuracy) and rsvd / rid
against the same blocks in a small batch (the other variants), and sizes on the
other side of the line.

Tolerances as in the operations' own tests: additions 1e-11 of the operands' norms
with equal ranks, rsvd / rid products 1e-10 of the block's norm."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("alg,eps", [("rounded_addition", 0.0), ("rounded_addition", 1e-6), ("fast_rounded_addition", 0.0)])
@pytest.mark.parametrize("m,n,ka,kb", [(24, 24, 3, 2), (64, 50, 8, 8), (17, 9, 8, 8), (128, 128, 8, 8), (129, 40, 8, 8),
                                       (256, 256, 4, 3), (64, 64, 9, 8)])
def test_lowrank_add_many(gpu_lib, alg, eps, m, n, ka, kb):
    import torch
    rng = np.random.default_rng(m + n + ka)
    count, few, kmax = 400, 5, min(ka + kb, m, n)
    q = lambda r, k: np.stack([np.linalg.qr(rng.standard_normal((r, k)))[0] for _ in range(count)])
    Ua0, Va0, Ub, Vb = q(m, ka), q(n, ka), q(m, kb), q(n, kb)
    Sa0, Sb = np.diag(0.6 ** np.arange(ka)), np.diag(0.5 ** np.arange(kb))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def add(c):
        U, S, V = np.zeros((c, kmax, m)), np.zeros((c, kmax, kmax)), np.zeros((c, n, kmax))
        U[:, :ka], S[:, :ka, :ka], V[:, :, :ka] = Ua0[:c].swapaxes(1, 2), Sa0, Va0[:c]
        dU, dS, dV = dev(U), dev(S), dev(V)
        dk = torch.full((c,), ka, dtype=torch.int32, device="cuda")
        db = torch.full((c,), kb, dtype=torch.int32, device="cuda")
        dUb, dSb, dVb = dev(Ub[:c].swapaxes(1, 2)), dev(np.stack([Sb] * c)), dev(Vb[:c])
        rc = gpu_lib.frank_lowrank_add_batched(m, n, c, kmax, alg.encode(), eps, _p(dU), m, m * kmax, _p(dS), kmax,
                                               kmax * kmax, _p(dV), kmax, kmax * n, _p(dk), _p(dUb), m, m * kb, _p(dSb),
                                               kb, kb * kb, _p(dVb), kb, kb * n, _p(db), kb, None)
        assert rc == 0, gpu_lib.frank_last_error()
        k = dk.cpu().numpy()
        return k, [dU[b, :k[b]].T.cpu().numpy() @ dS[b, :k[b], :k[b]].T.cpu().numpy() @ dV[b, :, :k[b]].T.cpu().numpy()
                   for b in range(c)]

    k1, one = add(few)
    k2, many = add(count)
    assert np.array_equal(k1, k2[:few])
    tol = 1e-11 * (np.linalg.norm(Sa0) + np.linalg.norm(Sb))
    for a, b in zip(one, many):
        np.testing.assert_allclose(b, a, rtol=0, atol=tol)
    if eps > 0.0:                                     # the sum itself, to the accuracy
        for b in range(0, count, 37):
            D = Ua0[b] @ Sa0 @ Va0[b].T + Ub[b] @ Sb @ Vb[b].T
            assert np.linalg.norm(many[b] - D) <= 10 * eps * np.linalg.norm(D)


@pytest.mark.parametrize("m,n,rank", [(40, 33, 4), (128, 128, 8), (130, 128, 8)])
def test_rsvd_and_rid_many(gpu_lib, m, n, rank):
    import torch
    rng = np.random.default_rng(m)
    count = 300
    A = np.stack([rng.standard_normal((m, rank)) @ np.diag(0.5 ** np.arange(rank)) @ rng.standard_normal((rank, n))
                  for _ in range(count)])
    dA = torch.from_numpy(np.ascontiguousarray(A.swapaxes(1, 2))).cuda()
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")
    for op in ("rsvd", "rid"):
        U, S, V = z(count, rank, m), z(count, rank, rank), z(count, n, rank)
        out = (_p(U), m, m * rank, _p(S), rank, rank * rank, _p(V), rank, rank * n, None)
        if op == "rsvd":
            rc = gpu_lib.frank_rsvd_batched(m, n, count, rank, 5, 1, _p(dA), m, m * n, *out)
        else:
            rc = gpu_lib.frank_rid_batched(m, n, count, rank + 5, rank, _p(dA), m, m * n, *out)
        assert rc == 0, gpu_lib.frank_last_error()
        got = (V @ S @ U).swapaxes(1, 2).cpu().numpy()       # column-major blocks: (U S V)^T = V^T S^T U^T
        for b in range(0, count, 23):
            assert np.linalg.norm(got[b] - A[b]) <= 1e-10 * np.linalg.norm(A[b]), (op, b)
