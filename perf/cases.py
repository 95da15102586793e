"""Performance cases of the factor-and-solve path, through the public entry points.

Each case is one piece of work that a user of the framework has it do: factor a
block low-rank (BLR) or hierarchical (H) kernel matrix and solve to a residual,
solve again with a kept factor, multiply, factor a batch of systems, run a
differentiable solve, or add low-rank blocks.  The `op` of a case says which:

  factor       A.getrf() + A.refine_device() on a kept BLR plan
  refine       A.refine_device() on a kept factor (new right-hand sides)
  matvec       A.matvec_device() (the FP64 H-matvec)
  hlu          H.getrf() + H.refine_device() on a kept H-matrix
  batch        BLRBatch.getrf() + refine_device() over independent systems
  adjoint      forward + backward of frank_b200.adjoint.solve_exp
  lowrank_add  LowRank += LowRank of a batch of blocks (per-operation C ABI)

Points are uniform in the unit cube (sorted in 1-D, Morton ordered in 2-D and
3-D), right-hand sides N(0, 1), as the framework's benchmark draws them.
"""
import ctypes
import math

import numpy as np
import torch

import frank_b200
from frank_b200 import BLRMatrix, HMatrix
from frank_b200.adjoint import solve_exp
from frank_b200.batch import BLRBatch


def listed():
    return [
        # the benchmark's headline: 3-D Laplace, 64 x 64 blocks of 512, FP32 factor + FP64 refinement
        # (ranks stay far below 384, so a program bounds the storage of its blocks there)
        dict(name="blr_mixed_n32768", op="factor", kernel="laplace", dim=3, n=32768, nb=64, prec="mixed",
             eps=1e-8, feps=3e-3, rank=0, max_rank=384, nrhs=4, tol=1e-10),
        # the same problem in plain FP64 at the accuracy of A_H, on the order of the framework's mid-size tests
        dict(name="blr_fp64_n8192", op="factor", kernel="laplace", dim=3, n=8192, nb=16, prec="fp64",
             eps=1e-8, feps=1e-8, rank=0, nrhs=4, tol=1e-12),
        # an order that no block size divides (blocks of 501, a last one of 496), odd right-hand sides
        dict(name="blr_mixed_ragged_n6007", op="factor", kernel="laplace", dim=2, n=6007, nb=12, prec="mixed",
             eps=1e-6, feps=1e-3, rank=0, nrhs=3, tol=1e-11),
        # fixed-rank BLR (the reference's default addition): 1-D Laplace, 8 x 8 blocks of 256, rank 16
        dict(name="blr_rank16_n2048", op="factor", kernel="laplace", dim=1, n=2048, nb=8, prec="fp64",
             eps=0.0, feps=0.0, rank=16, nrhs=1, tol=1e-12),
        # the smallest problems (the reference's test grid): blocks of 32, where latency counts
        dict(name="blr_fp64_n256", op="factor", kernel="laplace", dim=1, n=256, nb=8, prec="fp64",
             eps=1e-8, feps=1e-8, rank=0, nrhs=1, tol=1e-12),
        # new right-hand sides against a factor that is kept
        dict(name="blr_refine_n16384", op="refine", kernel="laplace", dim=3, n=16384, nb=32, prec="mixed",
             eps=1e-8, feps=3e-3, rank=0, nrhs=8, tol=1e-10),
        # the compressed matrix as an operator (iterative methods, residuals)
        dict(name="blr_matvec_n16384", op="matvec", kernel="laplace", dim=3, n=16384, nb=32, prec="fp64",
             eps=1e-8, feps=1e-8, rank=0, nrhs=4, tol=0.0),
        # multi-level H-LU at the benchmark's order: binary tree of 9 levels, leaves of 256, rank 32
        dict(name="hlu_n131072", op="hlu", kernel="laplace", dim=3, n=131072, leaf=256, rank=32, nrhs=8, tol=1e-10),
        # multi-level H-LU of a small 1-D problem (leaves of 64, rank 16)
        dict(name="hlu_n2048", op="hlu", kernel="laplace", dim=1, n=2048, leaf=64, rank=16, nrhs=1, tol=1e-12),
        # independent uneven systems, one launch per elimination step over all of them
        dict(name="batch_24", op="batch", kernel="neglog", dim=2, nmin=1024, nmax=4096, count=24, block=256,
             prec="mixed", eps=1e-6, feps=1e-4, grid=16, nrhs=1, tol=1e-10),
        # differentiable solve: construction, factorization, solve, adjoint solve, d/dtheta
        dict(name="adjoint_n4096", op="adjoint", kernel="exp", dim=2, n=4096, nb=8, prec="fp64",
             eps=1e-9, feps=1e-9, rank=0, nrhs=1, tol=1e-12, theta=0.2, nugget=1e-2),
        # block arithmetic one operation at a time: A += B on blocks of 256 of rank 32
        dict(name="lowrank_add_256", op="lowrank_add", m=256, k=32, count=16, lra="fast_rounded_addition"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["factor", "factor", "factor", "refine", "matvec", "hlu", "batch", "adjoint", "lowrank_add"])
    if op in ("factor", "refine", "matvec"):
        form = rng.choice(["mixed", "fp64", "rank"]) if op != "matvec" else "fp64"
        dim = rng.choice([2, 3])
        block = _log_int(rng, 32, 512)
        n = _log_int(rng, 4 * block, min(48 * block, 16384 if form == "mixed" else 8192))
        nb = max(2, -(-n // block))
        while (nb - 1) * -(-n // nb) >= n or n - (nb - 1) * -(-n // nb) < 24:   # no empty or sliver last block
            n += 1
        nrhs = rng.randint(1, 8)
        if form == "rank":
            return dict(op=op, kernel="laplace", dim=1, n=n, nb=nb, prec="fp64", eps=0.0, feps=0.0,
                        rank=rng.randint(4, 16), nrhs=nrhs, tol=1e-12)
        if form == "fp64":
            eps = 10.0 ** -rng.randint(6, 9)
            return dict(op=op, kernel="laplace", dim=dim, n=n, nb=nb, prec="fp64", eps=eps, feps=eps, rank=0,
                        nrhs=nrhs, tol=0.0 if op == "matvec" else 1e-12)
        return dict(op=op, kernel="laplace", dim=dim, n=n, nb=nb, prec="mixed", eps=10.0 ** -rng.randint(6, 8),
                    feps=rng.choice([3e-3, 1e-3, 1e-4]), rank=0, nrhs=nrhs, tol=1e-11)
    if op == "hlu":
        leaf = rng.randint(32, 256)
        levels = rng.randint(2, 7)
        return dict(op=op, kernel="laplace", dim=rng.choice([1, 3]), n=leaf << levels, leaf=leaf,
                    rank=rng.randint(4, min(32, leaf // 4)), nrhs=rng.randint(1, 8), tol=1e-10)
    if op == "batch":
        return dict(op=op, kernel="neglog", dim=2, nmin=512, nmax=_log_int(rng, 1024, 4096), count=rng.randint(4, 24),
                    block=rng.choice([128, 256]), prec="mixed", eps=1e-6, feps=1e-4, grid=rng.choice([8, 16]),
                    nrhs=rng.randint(1, 3), tol=1e-10)
    if op == "adjoint":
        n = _log_int(rng, 512, 4096)
        nb = max(2, n // rng.choice([128, 256, 512]))
        while (nb - 1) * -(-n // nb) >= n or n - (nb - 1) * -(-n // nb) < 24:
            n += 1
        return dict(op=op, kernel="exp", dim=2, n=n, nb=nb, prec="fp64", eps=1e-9, feps=1e-9, rank=0, nrhs=1,
                    tol=1e-12, theta=rng.uniform(0.15, 0.3), nugget=1e-2)
    k = rng.randint(4, 32)
    return dict(op=op, m=_log_int(rng, 3 * k, 1024), k=k, count=_log_int(rng, 1, 64),
                lra=rng.choice(["fast_rounded_addition", "rounded_addition"]))


# -- inputs ---------------------------------------------------------------------

def _points(n, dim, rng):
    x = rng.random((dim, n))
    if dim == 1:
        return np.sort(x, axis=1)
    level = 20 if dim == 2 else 16
    ix = (x * (1 << level)).astype(np.int64)
    code = np.zeros(n, dtype=np.int64)
    for lev in range(level):
        for d in range(dim):
            code |= ((ix[d] >> lev) & 1) << (dim * lev + d)
    return np.ascontiguousarray(x[:, np.argsort(code, kind="stable")])


def _rhs(n, nrhs, rng):
    """nrhs x n, i.e. the column-major n x nrhs block the device entry points take."""
    return torch.from_numpy(rng.standard_normal((nrhs, n))).cuda()


def _batch_sizes(case, rng):
    b = case["block"]
    return [b * int(k) for k in rng.integers(max(2, case["nmin"] // b), case["nmax"] // b + 1, size=case["count"])]


def _blocks(case, rng):
    """Low-rank blocks: left and right orthonormal bases, singular values over six decades."""
    m, k, c = case["m"], case["k"], case["count"]
    out = []
    for _ in range(2):
        U = np.linalg.qr(rng.standard_normal((c, m, k)))[0]
        V = np.linalg.qr(rng.standard_normal((c, m, k)))[0]
        s = 10.0 ** -np.sort(rng.uniform(0.0, 6.0, (c, k)), axis=1)
        out.append((U, s, V))
    return out


def _plan(case, pts):
    M = BLRMatrix(case["n"], case["nb"], eps=case["feps"], fixed_rank=case["rank"], precision=case["prec"],
                  max_rank=case.get("max_rank", 0))
    M.build_kernel(case["kernel"], pts, case["eps"])
    return M


class _State:
    pass


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    s.case, op = case, case["op"]
    if op in ("factor", "refine", "matvec"):
        s.M = _plan(case, _points(case["n"], case["dim"], rng))
        s.b = _rhs(case["n"], case["nrhs"], rng)
        s.x = torch.zeros_like(s.b)
        if op == "refine":
            s.M.getrf()
    elif op == "hlu":
        s.M = HMatrix(case["n"], case["leaf"], case["rank"])
        s.M.build_kernel(case["kernel"], _points(case["n"], case["dim"], rng))
        s.b = _rhs(case["n"], case["nrhs"], rng)
        s.x = torch.zeros_like(s.b)
    elif op == "batch":
        s.sizes = _batch_sizes(case, rng)
        s.plans = []
        for n in s.sizes:
            M = BLRMatrix(n, n // case["block"], eps=case["feps"], precision=case["prec"], max_rank=96)
            M.build_kernel(case["kernel"], _points(n, case["dim"], rng), case["eps"], params=(float(n),))
            s.plans.append(M)
        s.batch = BLRBatch(s.plans, grid=case["grid"])
        s.ld = max(s.sizes)
        s.b = torch.zeros((len(s.sizes), case["nrhs"], s.ld), dtype=torch.float64, device="cuda")
        for k, n in enumerate(s.sizes):
            s.b[k, :, :n] = _rhs(n, case["nrhs"], rng)
        s.x = torch.zeros_like(s.b)
    elif op == "adjoint":
        s.pts = torch.from_numpy(_points(case["n"], case["dim"], rng))
        s.b = _rhs(case["n"], 1, rng)[0]
    else:
        (Ua, sa, Va), (Ub, sb, Vb) = _blocks(case, rng)
        # column-major blocks: U (m x kmax, ld m), S (kmax x kmax), V (kmax x m, ld kmax), kmax = k
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        s.Ua, s.Va, s.Ub, s.Vb = dev(Ua.swapaxes(1, 2)), dev(Va), dev(Ub.swapaxes(1, 2)), dev(Vb)
        s.Sa, s.Sb = torch.diag_embed(dev(sa)), torch.diag_embed(dev(sb))
        s.ka = torch.full((case["count"],), case["k"], dtype=torch.int32, device="cuda")
        s.kb = s.ka.clone()
    torch.cuda.synchronize()
    return s


def run(s):
    case, op = s.case, s.case["op"]
    if op == "matvec":
        s.M.matvec_device(s.b.data_ptr(), s.x.data_ptr(), case["nrhs"])
        return s.x
    if op in ("factor", "refine", "hlu"):
        if op != "refine":
            s.M.getrf()
        s.M.refine_device(s.b.data_ptr(), s.x.data_ptr(), case["nrhs"], tol=case["tol"], maxit=60)
        return s.x
    if op == "batch":
        s.batch.getrf()
        K = len(s.sizes)
        s.batch.refine_device([s.b[k].data_ptr() for k in range(K)], [s.x[k].data_ptr() for k in range(K)], s.ld,
                              case["nrhs"], tol=case["tol"])
        return s.x
    if op == "adjoint":
        b = s.b.clone().requires_grad_(True)
        th = torch.tensor(case["theta"], dtype=torch.float64, device="cuda", requires_grad=True)
        x = solve_exp(b, th, s.pts, case["nb"], eps=case["eps"], nugget=case["nugget"], precision=case["prec"],
                      factor_eps=case["feps"], tol=case["tol"])
        (0.5 * (x * x).sum()).backward()
        return [x.detach(), b.grad, th.grad]
    # the addition works in place on A: a caller that keeps the old block copies it first
    U, S, V, ka = s.Ua.clone(), s.Sa.clone(), s.Va.clone(), s.ka.clone()
    m, k = case["m"], case["k"]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = frank_b200.lib().frank_lowrank_add_batched(
        m, m, case["count"], k, case["lra"].encode(), 0.0, p(U), m, m * k, p(S), k, k * k, p(V), k, k * m, p(ka),
        p(s.Ub), m, m * k, p(s.Sb), k, k * k, p(s.Vb), k, k * m, p(s.kb), k, None)
    if rc != 0:
        raise RuntimeError(frank_b200.lib().frank_last_error().decode())
    # the bases are unique up to signs only: the block itself (transposed) and its singular values
    return [V @ S @ U, torch.diagonal(S, dim1=1, dim2=2), ka]


# -- what a pass cannot do without -------------------------------------------------

def _mean_rank(case):
    """Typical rank of a block at the factor's tolerance (fixed-rank plans: the rank)."""
    if case.get("rank"):
        return case["rank"]
    digits = -math.log10(case["feps"])
    return {1: 1.6 * digits, 2: 0.45 * digits ** 2 + 2, 3: 1.1 * digits ** 2 + 4}[case["dim"]]


def _blr_work(n, nb, r, elem, solves, nrhs, factor=True):
    b, pairs = n / nb, nb * (nb - 1)
    r = min(r, b / 2)
    size = nb * b * b + pairs * (2 * b * r + r * r)          # values of the matrix
    fl = solves * nrhs * 4.0 * size
    by = solves * size * (8 + elem) + 16.0 * n * nrhs
    if factor:
        steps = sum(m * (m - 1) for m in range(1, nb))        # low-rank additions
        dense = sum(m for m in range(1, nb))                  # dense updates
        fl += nb * 2 / 3 * b ** 3 + pairs * b * b * r + dense * 4 * b * b * r + steps * (30 * b * r * r + 80 * r ** 3)
        by += size * (8 + elem)
    return fl, by


def work(case):
    op = case["op"]
    elem = 4 if case.get("prec") == "mixed" else 8
    if op == "matvec":
        fl, by = _blr_work(case["n"], case["nb"], _mean_rank(case), 0, 0.5, case["nrhs"], factor=False)
        return {"bytes": 2 * by - 16 * case["n"] * case["nrhs"], "flops": fl}
    if op in ("factor", "refine"):
        solves = 5 if case["prec"] == "mixed" else 2
        fl, by = _blr_work(case["n"], case["nb"], _mean_rank(case), elem, solves, case["nrhs"], op == "factor")
        return {"bytes": by, "flops": fl}
    if op == "hlu":
        n, b, k = case["n"], case["leaf"], case["rank"]
        L = int(round(math.log2(n / b)))
        size = n * b + 2 * L * n * k
        # leaf LU and inverses, substitutions of the bases, additions (level l: every update of an ancestor)
        fl = n / b * 2 * b ** 3 + L * n * k * (2 * b + 4 * L * k) + L * (L - 1) / 2 * n * 30 * k * k
        return {"bytes": 16.0 * size + 5 * 16.0 * size, "flops": fl + 5 * 4.0 * size * case["nrhs"]}
    if op == "batch":
        n = (case["nmin"] + case["nmax"]) / 2
        fl, by = _blr_work(n, int(n // case["block"]), _mean_rank(case), elem, 4, case["nrhs"])
        return {"bytes": by * case["count"], "flops": fl * case["count"]}
    if op == "adjoint":
        fl, by = _blr_work(case["n"], case["nb"], _mean_rank(case), elem, 4, 1)
        b, pairs, r = case["n"] / case["nb"], case["nb"] * (case["nb"] - 1), _mean_rank(case)
        return {"bytes": by, "flops": fl + pairs * 4 * b * b * min(r, b) + 20.0 * case["n"] ** 2}
    m, k, c = case["m"], case["k"], case["count"]
    return {"bytes": 8.0 * c * 3 * (2 * m * k + k * k), "flops": c * (24.0 * m * k * k + 26 * (2 * k) ** 3)}


# -- the same results in plain 64-bit torch / numpy -----------------------------------

def _kernel(case, x, y, diag=0.0):
    """Kernel values between point sets x (dim x m) and y (dim x n)."""
    r = torch.zeros((x.shape[1], y.shape[1]), dtype=torch.float64, device=x.device)
    for d in range(x.shape[0]):
        r += (x[d][:, None] - y[d][None, :]) ** 2
    r = r.sqrt_()
    if case["kernel"] == "laplace":
        return r.add_(1e-3).reciprocal_()
    if case["kernel"] == "neglog":
        return r.add_(1e-3).log_().neg_()
    return r.mul_(-1.0 / case["theta"]).exp_()


def _omega(n, s):
    """n x s uniform [0, 1) values of a 32-bit Mersenne twister seeded 0, two draws a value, row by row."""
    bg = np.random.RandomState(0)
    raw = bg.randint(0, 1 << 32, size=2 * n * s, dtype=np.uint32).astype(np.float64)
    return torch.from_numpy(((raw[0::2] + raw[1::2] * 4294967296.0) / 18446744073709551616.0).reshape(n, s))


def _low_rank(A, k):
    """Rank-k approximation of A from the range of A Omega (k + 5 samples)."""
    s = min(k + 5, A.shape[0], A.shape[1])
    Q = torch.linalg.qr(A @ _omega(A.shape[1], s).to(A.device))[0]
    U, S, Vt = torch.linalg.svd(Q.T @ A, full_matrices=False)
    return (Q @ U[:, :k] * S[:k]) @ Vt[:k]


def exact(case, seed):
    rng = np.random.default_rng(seed)
    op = case["op"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if op == "hlu" and case["n"] > 32768:
        return None                                             # the dense matrix does not fit
    if op in ("factor", "refine", "matvec", "hlu"):
        n = case["n"]
        x = torch.from_numpy(_points(n, case["dim"], rng)).to(dev)
        b = torch.from_numpy(rng.standard_normal((case["nrhs"], n))).to(dev)
        A = _kernel(case, x, x)
        if op == "hlu":
            size = n // 2
            while size >= case["leaf"]:
                for c in range(n // size):
                    i, j = c * size, (c ^ 1) * size
                    A[i:i + size, j:j + size] = _low_rank(A[i:i + size, j:j + size].clone(), case["rank"])
                size //= 2
        elif case["rank"]:
            step = -(-n // case["nb"])
            for i in range(0, n, step):
                for j in range(0, n, step):
                    if i != j:
                        A[i:i + step, j:j + step] = _low_rank(A[i:i + step, j:j + step].clone(), case["rank"])
        return (A @ b.T).T.contiguous() if op == "matvec" else torch.linalg.solve(A, b.T).T.contiguous()
    if op == "batch":
        sizes = _batch_sizes(case, rng)
        pts = [_points(n, case["dim"], rng) for n in sizes]
        out = torch.zeros((len(sizes), case["nrhs"], max(sizes)), dtype=torch.float64, device=dev)
        for k, n in enumerate(sizes):
            x = torch.from_numpy(pts[k]).to(dev)
            A = _kernel(case, x, x)
            A.diagonal().add_(float(n))
            b = torch.from_numpy(rng.standard_normal((case["nrhs"], n))).to(dev)
            out[k, :, :n] = torch.linalg.solve(A, b.T).T
        return out
    if op == "adjoint":
        x = torch.from_numpy(_points(case["n"], case["dim"], rng)).to(dev)
        b = torch.from_numpy(rng.standard_normal((1, case["n"]))).to(dev)[0]
        K = _kernel(case, x, x)
        A = K.clone()
        A.diagonal().add_(case["nugget"])
        sol = torch.linalg.solve(A, b)
        lam = torch.linalg.solve(A.T, sol)
        dK = K * (-K.log()) / case["theta"]                   # exp(-r/theta) r / theta^2
        return [sol, lam, -(lam @ (dK @ sol))]
    (Ua, sa, Va), (Ub, sb, Vb) = _blocks(case, rng)
    D = (Ua * sa[:, None, :]) @ Va.swapaxes(1, 2) + (Ub * sb[:, None, :]) @ Vb.swapaxes(1, 2)
    D = torch.from_numpy(D).to(dev)
    U, S, Vt = torch.linalg.svd(D, full_matrices=False)
    k = case["k"]
    best = (U[:, :, :k] * S[:, None, :k]) @ Vt[:, :k]
    return [best.transpose(1, 2).contiguous(), S[:, :k].contiguous(), None]
