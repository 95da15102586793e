// Cooperative FP64 building blocks for a group of warps of one CTA: all of it,
// or one half while the other half works on something independent (the U and
// the V side of a low-rank block).  A group synchronises on its own named
// barrier.  Matrices are column-major; a pointer may be shared or global
// memory.  Every routine is called by all threads of the group and ends with
// the group's barrier.
//
// What bounds these routines is latency, not work (a target of the headline
// factorization is a few MFLOP): so the products read their tensor-pipe
// fragments where they lie, the column steps of the factorizations take one
// barrier each, and columns belong to groups of lanes rather than warps where
// they are short, which makes a reduction three exchanges instead of five and
// puts four columns into flight per warp.
#pragma once

namespace frank {

struct Grp {
  int tid, nt, wid, nw, bar;
  FRANK_D void sync() const {
    if (bar == 0) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nt) : "memory");
  }
};

FRANK_D Grp grp_all() {
  return Grp{(int)threadIdx.x, (int)blockDim.x, (int)(threadIdx.x >> 5), (int)(blockDim.x >> 5), 0};
}
// Half h (0, 1) of the CTA; blockDim.x a multiple of 64.
FRANK_D Grp grp_half(int h) {
  const int nt = blockDim.x / 2;
  return Grp{(int)threadIdx.x - h * nt, nt, (int)(threadIdx.x - h * nt) >> 5, nt >> 5, 1 + h};
}

// Shared memory of a group's factorizations.
constexpr int GQ = 32;   // widest panel
struct GrpShared {
  double G[GQ * GQ];     // V^T V of a panel (strictly upper part)
  double T[GQ * GQ];     // its T factor
  double tau[GQ], beta[GQ], scal[GQ];
  double part[8 * 64];   // partial tiles of short products
};

// C (m x n) = alpha op(A) op(B) + beta C as cta_gemm, on the group's warps.  An output
// of at most four 8 x 8 tiles splits a long inner dimension over eight warps;
// the split depends on the shape only, so a result does not depend on the
// group's size.  part: 8 * 64 doubles.
template <typename TA, typename TB, typename TC>
static __device__ __noinline__ void g_gemm(Grp g, int m, int n, int k, double alpha, const TA* A, int64_t lda, bool ta,
                                    const TB* B, int64_t ldb, bool tb, double beta, TC* C, int64_t ldc,
                                    double* part) {
  if (m <= 0 || n <= 0) { g.sync(); return; }
  const int lane = threadIdx.x & 31;
  const int64_t sai = ta ? lda : 1, sak = ta ? 1 : lda, sbj = tb ? 1 : ldb, sbk = tb ? ldb : 1;
  const int tm = (m + 7) / 8, t8 = tm * ((n + 7) / 8);
  if (t8 <= 4 && k >= 64 && g.nw >= 8) {
    const int split = 8 / t8, kc = ((k + split - 1) / split + 3) & ~3;
    const int tile = g.wid / split, q = g.wid % split;
    if (tile < t8) {
      double acc[1][1][2];
      warp_dgemm_acc<1, 1>(m, n, min(k, q * kc), min(k, (q + 1) * kc), A, sai, sak, B, sbj, sbk, (tile % tm) * 8,
                           (tile / tm) * 8, acc);
      part[g.wid * 64 + 2 * lane] = acc[0][0][0];
      part[g.wid * 64 + 2 * lane + 1] = acc[0][0][1];
    }
    g.sync();
    for (int e = g.tid; e < t8 * 64; e += g.nt) {
      const int tl = e >> 6, x = e & 63;
      const int r = (tl % tm) * 8 + (x >> 3), c = (tl / tm) * 8 + (x & 7);
      if (r < m && c < n) {
        double v = 0.0;
        for (int s = 0; s < split; ++s) v += part[(tl * split + s) * 64 + x];
        dgemm_store(C + r + (int64_t)c * ldc, v, alpha, beta);
      }
    }
    g.sync();
    return;
  }
  auto cost = [&](int mi, int ni) {
    const int tiles = ((m + 8 * mi - 1) / (8 * mi)) * ((n + 8 * ni - 1) / (8 * ni));
    return ((tiles + g.nw - 1) / g.nw) * (2 * mi * ni + mi + ni);
  };
  const int c23 = cost(2, 3), c42 = cost(4, 2), c22 = cost(2, 2), c11 = cost(1, 1);
  const int best = min(min(c23, c42), min(c22, c11));
  if (best == c23)
    warps_dgemm<2, 3>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  else if (best == c42)
    warps_dgemm<4, 2>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  else if (best == c22)
    warps_dgemm<2, 2>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  else
    warps_dgemm<1, 1>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  g.sync();
}

// C (m x n, ldc) = alpha A^T B over k rows, A (k x m, lda), B (k x n, ldb), k
// long: every warp takes an eighth of the rows for 24 x 24 tiles of C, so that
// each row of A and B is read once per tile and all warps have equal work; the
// eight partial products go to part (in L2; G_TN_PART doubles) and are summed in
// order.  Outputs above G_TN_TILES 8 x 8 tiles take g_gemm (they fill the
// warps by themselves).
constexpr int G_TN_TILES = 81;
constexpr int G_TN_PART = 8 * 72 * 72;

template <typename TA, typename TB>
static __device__ __noinline__ void g_gemm_tn(Grp g, int m, int n, int k, double alpha, const TA* A, int64_t lda, const TB* B,
                                       int64_t ldb, double* C, int64_t ldc, double* part, double* spart) {
  const int m8 = (m + 7) / 8, n8 = (n + 7) / 8;
  if (m8 * n8 > G_TN_TILES || m8 > 9 || n8 > 9 || k < 128 || g.nw < 8) {
    g_gemm(g, m, n, k, alpha, A, lda, true, B, ldb, false, 0.0, C, ldc, spart);
    return;
  }
  const int lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
  const int kc = ((k + 7) / 8 + 3) & ~3, q = g.wid & 7, sub = g.wid >> 3, nsub = g.nw >> 3;
  const int k0 = min(k, q * kc), k1 = min(k, k0 + kc);
  const int tm = (m8 + 2) / 3, tn = (n8 + 2) / 3, mp = tm * 24;
  double* pq = part + (int64_t)q * mp * tn * 24;
  for (int tile = sub; tile < tm * tn; tile += nsub) {
    const int i0 = (tile % tm) * 24, j0 = (tile / tm) * 24;
    double acc[3][3][2];
    warp_dgemm_acc<3, 3>(m, n, k0, k1, A, lda, 1, B, ldb, 1, i0, j0, acc);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        pq[(i0 + 8 * i + gr) + (int64_t)(j0 + 8 * j + 2 * t) * mp] = acc[i][j][0];
        pq[(i0 + 8 * i + gr) + (int64_t)(j0 + 8 * j + 2 * t + 1) * mp] = acc[i][j][1];
      }
  }
  g.sync();
  for (int e = g.tid; e < m * n; e += g.nt) {
    const int r = e % m, c = e / m;
    const double* p = part + r + (int64_t)c * mp;
    double v[8], s = 0.0;
#pragma unroll
    for (int x = 0; x < 8; ++x) v[x] = p[(int64_t)x * mp * tn * 24];
#pragma unroll
    for (int x = 0; x < 8; ++x) s += v[x];
    C[r + (int64_t)c * ldc] = alpha * s;
  }
  g.sync();
}

// Sums of v[0..N) over the warp (every lane gets them).
template <int N>
FRANK_D void warp_sums(double (&v)[N]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

// Householder quantities (dlarfg) of a column with leading entry alpha and
// squared norm xn2 below it.
FRANK_D void reflector(double alpha, double xn2, double& beta, double& tau, double& scal) {
  if (xn2 > 0.0) {
    const double nrm = sqrt(alpha * alpha + xn2);
    beta = alpha >= 0.0 ? -nrm : nrm;
    tau = (beta - alpha) / beta;
    scal = 1.0 / (alpha - beta);
  } else {
    beta = alpha;
    tau = 0.0;
    scal = 0.0;
  }
}

// Householder QR (dgeqr2 conventions) of a panel P (m x n, ldp, n <= GQ, in
// shared memory).  One barrier per column: every warp that updates columns
// forms the reflector itself from the column it reads anyway, and reflectors
// stay unscaled until the end.  The dot products of each reflector with the
// earlier ones are formed in the same pass by the same warps, so the T factor
// needs no product of its own.  On return P holds the clean V (unit lower
// trapezoid), s.T the T factor (upper, zero below), s.tau; R (min(m, n) x n)
// goes to R (ldr) with zeros below its diagonal.
static __device__ __noinline__ void g_panel_qr(Grp g, int m, int n, double* P, int ldp, double* R, int64_t ldr,
                                        GrpShared& s) {
  const int lane = threadIdx.x & 31, km = min(m, n);
  for (int j = 0; j < km; ++j) {
    const double* x = P + (int64_t)j * ldp;
    const double alpha = x[j];
    // columns c != j of this warp: c = wid, wid + nw, ...; c > j updated, c < j dots only
    double xn2 = 0.0, beta = 0.0, tau = 0.0, scal = 0.0;
    bool have = false;
    for (int c0 = g.wid; c0 < n; c0 += 4 * g.nw) {
      double* p[4];
      double d[5];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = c0 + i * g.nw;
        p[i] = P + (int64_t)(c < n && c != j ? c : j) * ldp;
        d[i] = 0.0;
      }
      d[4] = 0.0;
      const int cnt = min(4, (n - c0 + g.nw - 1) / g.nw);
      if (cnt > 2) {
#pragma unroll 4
        for (int e = j + 1 + lane; e < m; e += 32) {
          const double v = x[e];
          d[4] = fma(v, v, d[4]);
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] = fma(v, p[i][e], d[i]);
        }
        warp_sums<5>(d);
      } else {
#pragma unroll 4
        for (int e = j + 1 + lane; e < m; e += 32) {
          const double v = x[e];
          d[4] = fma(v, v, d[4]);
          d[0] = fma(v, p[0][e], d[0]);
          d[1] = fma(v, p[1][e], d[1]);
        }
        double h[3] = {d[0], d[1], d[4]};
        warp_sums<3>(h);
        d[0] = h[0]; d[1] = h[1]; d[4] = h[2];
      }
      if (!have) {
        xn2 = d[4];
        reflector(alpha, xn2, beta, tau, scal);
        have = true;
      }
      double f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = c0 + i * g.nw;
        f[i] = 0.0;
        if (c >= n) continue;
        if (c > j) {
          const double top = p[i][j], w = tau * fma(scal, d[i], top);
          f[i] = w * scal;
          __syncwarp();
          if (lane == 0) p[i][j] = top - w;
        } else if (c < j) {
          // v_c . v_j: rows below j of both, and row j where v_j is 1
          if (lane == 0) s.G[c + j * GQ] = s.scal[c] * fma(scal, d[i], p[i][j]);
        } else if (lane == 0) {
          s.tau[j] = tau; s.beta[j] = beta; s.scal[j] = scal;
        }
      }
      if (tau != 0.0) {
        const bool two = c0 + 2 * g.nw < n && c0 + (cnt - 1) * g.nw > j;
        if (two) {
#pragma unroll 4
          for (int e = j + 1 + lane; e < m; e += 32) {
            const double v = x[e];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (f[i] != 0.0) p[i][e] = fma(-f[i], v, p[i][e]);
          }
        } else if (f[0] != 0.0 || f[1] != 0.0) {
#pragma unroll 4
          for (int e = j + 1 + lane; e < m; e += 32) {
            const double v = x[e];
            if (f[0] != 0.0) p[0][e] = fma(-f[0], v, p[0][e]);
            if (f[1] != 0.0) p[1][e] = fma(-f[1], v, p[1][e]);
          }
        }
      }
    }
    g.sync();
  }
  // T = (triu(G, 1) + diag(1 / tau))^{-1}: lane = row, a column per warp and
  // pass, back substitution with the solved value by shuffle (tau_s multiplies
  // where the inverse would divide; tau = 0 gives a zero row and column)
  {
    const double tr = lane < km ? s.tau[lane] : 0.0;
    for (int c = g.wid; c < km; c += g.nw) {
      double up = lane == c ? 1.0 : 0.0;
      for (int q = c; q >= 0; --q) {
        const double xq = __shfl_sync(0xffffffffu, up * tr, q);
        if (lane < q) up = fma(-s.G[lane + q * GQ], xq, up);
        else if (lane == q) up = xq;
      }
      s.T[lane + c * GQ] = lane <= c ? up : 0.0;
    }
  }
  // R out, clean V in place
  for (int c = g.wid; c < n; c += g.nw) {
    double* pc = P + (int64_t)c * ldp;
    const double b = c < km ? s.beta[c] : 0.0, sc = c < km ? s.scal[c] : 0.0;
    for (int e = lane; e < km; e += 32) R[e + (int64_t)c * ldr] = e < c ? pc[e] : (e == c ? b : 0.0);
    __syncwarp();
    if (c < km)
      for (int e = lane; e < m; e += 32) pc[e] = e > c ? pc[e] * sc : (e == c ? 1.0 : 0.0);
  }
  g.sync();
}

FRANK_HD int panel_ld(int m) { return ((m + 15) & ~15) + 4; }   // 4 mod 16: conflict-free fragments

// Scratch of the blocked routines: W, W2 (GQ x widest operand each) and the
// partial products, in global memory.
struct GrpScratch {
  double *W, *W2, *part;
};

// Blocked Householder QR of A (m x n, lda): panels of w <= GQ columns in smP
// (panel_ld(m) x w doubles, shared), T factors in Tf (GQ x GQ per panel), the
// clean V of each panel left in A (rows and columns j0 ..), R (min(m, n) x n,
// ldr, zeros below the diagonal) apart.
static __device__ __noinline__ void g_qr(Grp g, int m, int n, double* A, int64_t lda, double* R, int64_t ldr, double* Tf,
                                  int w, double* smP, GrpShared& s, GrpScratch x) {
  const int km = min(m, n), ldp = panel_ld(m);
  for (int j0 = 0, p = 0; j0 < km; j0 += w, ++p) {
    const int jn = min(w, km - j0), mr = m - j0;
    double* Ap = A + j0 + (int64_t)j0 * lda;
    const int lane = threadIdx.x & 31;
    for (int c = g.wid; c < jn; c += g.nw)
#pragma unroll 4
      for (int r = lane; r < mr; r += 32) smP[r + c * ldp] = Ap[r + (int64_t)c * lda];
    // R rows below this panel's diagonal block are zero
    for (int c = g.wid; c < jn; c += g.nw)
      for (int r = j0 + jn + lane; r < km; r += 32) R[r + (int64_t)(j0 + c) * ldr] = 0.0;
    g.sync();
    g_panel_qr(g, mr, jn, smP, ldp, R + j0 + (int64_t)j0 * ldr, ldr, s);
    for (int c = g.wid; c < jn; c += g.nw)
#pragma unroll 4
      for (int r = lane; r < mr; r += 32) Ap[r + (int64_t)c * lda] = smP[r + c * ldp];
    for (int e = g.tid; e < GQ * GQ; e += g.nt) Tf[(int64_t)p * GQ * GQ + e] = s.T[e];
    const int nc = n - j0 - jn;
    if (nc > 0) {
      double* At = A + j0 + (int64_t)(j0 + jn) * lda;
      g_gemm_tn(g, jn, nc, mr, 1.0, smP, ldp, At, lda, x.W, GQ, x.part, s.part);
      g_gemm(g, jn, nc, jn, 1.0, s.T, GQ, true, x.W, GQ, false, 0.0, x.W2, GQ, s.part);
      g_gemm(g, mr, nc, jn, -1.0, smP, ldp, false, x.W2, GQ, false, 1.0, At, lda, s.part);
      // the finished rows of R
      for (int e = g.tid; e < jn * nc; e += g.nt) {
        const int r = e % jn, c = e / jn;
        R[(j0 + r) + (int64_t)(j0 + jn + c) * ldr] = At[r + (int64_t)c * lda];
      }
    }
    g.sync();
  }
}

// X (m x r, ldx) := Q X with the k reflectors of g_qr (clean V in A, Tf, panels
// of w).  Rows of X at or below nz are zero on entry.
static __device__ __noinline__ void g_apply_q(Grp g, int m, int k, const double* A, int64_t lda, const double* Tf, int w,
                                       int r, double* X, int64_t ldx, int nz, GrpShared& s, GrpScratch x) {
  for (int p = (k + w - 1) / w - 1; p >= 0; --p) {
    const int j0 = p * w, jn = min(w, k - j0), mr = m - j0;
    const int kr = min(mr, max(0, nz - j0));
    nz = m;
    if (kr == 0) continue;
    const double* V = A + j0 + (int64_t)j0 * lda;
    const double* T = Tf + (int64_t)p * GQ * GQ;
    g_gemm_tn(g, jn, r, kr, 1.0, V, lda, X + j0, ldx, x.W, GQ, x.part, s.part);
    g_gemm(g, jn, r, jn, 1.0, T, GQ, false, x.W, GQ, false, 0.0, x.W2, GQ, s.part);
    g_gemm(g, mr, r, jn, -1.0, V, lda, false, x.W2, GQ, false, 1.0, X + j0, ldx, s.part);
  }
}

// Project the columns of Y (m x p, ldy) out of the span of Q (m x k, ldq,
// orthonormal columns), twice (classical Gram-Schmidt with one
// re-orthogonalisation): Z (k x p, ldz) = Q^T Y_0, Y = (I - Q Q^T)^2 Y_0,
// Y_0 = Q Z + Y.  Z2 (k x p) is scratch.
template <typename T>
FRANK_D void g_project_out(Grp g, int m, int k, int p, const T* Q, int64_t ldq, double* Y, int64_t ldy, double* Z,
                           int64_t ldz, double* Z2, GrpShared& s, GrpScratch x) {
  for (int pass = 0; pass < 2; ++pass) {
    double* Zp = pass ? Z2 : Z;
    const int64_t ldp = pass ? k : ldz;
    g_gemm_tn(g, k, p, m, 1.0, Q, ldq, Y, ldy, Zp, ldp, x.part, s.part);
    g_gemm(g, m, p, k, -1.0, Q, ldq, false, Zp, ldp, false, 1.0, Y, ldy, s.part);
  }
  for (int e = g.tid; e < k * p; e += g.nt) Z[(e % k) + (int64_t)(e / k) * ldz] += Z2[e];
  g.sync();
}

// Largest key of the lanes with ties toward the smallest index (keys are
// non-negative; idx < 0: none).
FRANK_D void warp_argmax_key(double& v, int& idx) {
  const unsigned hi = idx < 0 ? 0u : (unsigned)__double2hiint(v), lo = idx < 0 ? 0u : (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const unsigned mi = __reduce_min_sync(0xffffffffu, idx >= 0 && hi == mh && lo == ml ? (unsigned)idx : ~0u);
  v = __hiloint2double((int)mh, (int)ml);
  idx = (int)mi;
}

// Truncated column-pivoted Householder QR of A (m x n, lda, shared memory)
// with the pivots and the stopping rule of truncated_geqp3
// (operations/LAPACK/geqp3.cpp:71-192): stop when the largest remaining
// column norm is at most thr, or after maxr steps.  A column belongs to eight
// lanes, columns stay where they are, every step takes one barrier: each warp
// reads the pivot column, forms the reflector itself, and updates its columns
// and their remaining norms (recomputed, not down-dated) in one pass.  On
// return ord[j] is the column chosen at step j, at[c] the step that chose
// column c (or m + n), tau[j]; column ord[j] holds R above row j, R(j, j) at
// row j and the scaled reflector below; every other column its rows of R.
// cand: 4 * nw doubles (two rows of values and indices); vec: 2 min(m, n)
// doubles.  All shared.
static __device__ __noinline__ int g_rrqr(Grp g, int m, int n, double* A, int lda, double thr, int maxr, double* tau,
                                   int* ord, int* at, double* vec, double* cand) {
  const int lane = threadIdx.x & 31, sub = lane >> 3, l8 = lane & 7;
  const int mind = min(min(m, n), maxr);
  double* scal = vec;
  double* beta = vec + min(m, n);
  const int ng = 4 * g.nw, gi = 4 * g.wid + sub;   // lane groups
  const double thr2 = thr >= 0.0 ? thr * thr : -1.0;
  double bv = -1.0;
  int bi = -1;
  for (int c0 = 0; c0 < n; c0 += ng) {
    const int c = c0 + gi;
    const double* p = A + (int64_t)min(c, n - 1) * lda;
    double q = 0.0;
    for (int e = l8; e < m; e += 8) q = fma(p[e], p[e], q);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (c < n) {
      if (l8 == 0) at[c] = m + n;
      if (q > bv) { bv = q; bi = c; }
    }
  }
  warp_argmax_key(bv, bi);
  double* cv = cand;
  int* ci = reinterpret_cast<int*>(cand + g.nw);
  if (lane == 0) { cv[g.wid] = bv; ci[g.wid] = bi; }
  g.sync();
  int r = 0;
  for (;;) {
    double mx = lane < g.nw ? cv[lane] : 0.0;
    int kp = lane < g.nw ? ci[lane] : -1;
    warp_argmax_key(mx, kp);
    if (r >= mind || kp < 0 || !(mx > thr2)) break;
    const double* x = A + (int64_t)kp * lda;
    const double alpha = x[r];
    double xn2 = 0.0, bt = 0.0, t = 0.0, sc = 0.0;
    bool have = false;
    bv = -1.0;
    bi = -1;
    for (int c0 = 0; c0 < n; c0 += ng) {
      const int c = c0 + gi;
      const bool live = c < n && c != kp && at[min(c, n - 1)] > r;
      double* p = A + (int64_t)min(c, n - 1) * lda;
      double d0 = 0.0, d1 = 0.0;
      if (!have) {
#pragma unroll 4
        for (int e = r + 1 + l8; e < m; e += 8) {
          const double v = x[e];
          d1 = fma(v, v, d1);
          d0 = fma(v, p[e], d0);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          d0 += __shfl_xor_sync(0xffffffffu, d0, o);
          d1 += __shfl_xor_sync(0xffffffffu, d1, o);
        }
        xn2 = d1;
        reflector(alpha, xn2, bt, t, sc);
        have = true;
      } else {
#pragma unroll 4
        for (int e = r + 1 + l8; e < m; e += 8) d0 = fma(x[e], p[e], d0);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) d0 += __shfl_xor_sync(0xffffffffu, d0, o);
      }
      const double top = p[r], w = live ? t * fma(sc, d0, top) : 0.0, f = w * sc;
      __syncwarp();
      double q = 0.0;
      if (live) {
        if (l8 == 0) p[r] = top - w;
#pragma unroll 4
        for (int e = r + 1 + l8; e < m; e += 8) {
          const double v = fma(-f, x[e], p[e]);
          p[e] = v;
          q = fma(v, v, q);
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (live && q > bv) { bv = q; bi = c; }
      if (c == kp && l8 == 0) {
        at[c] = r; ord[r] = c; tau[r] = t; beta[r] = bt; scal[r] = sc;
      }
    }
    warp_argmax_key(bv, bi);
    // the candidates of the previous step were read before this step's work,
    // but by warps that may still be at it: alternate two rows
    cv = cand + (r & 1 ? 0 : 2 * g.nw);
    ci = reinterpret_cast<int*>(cv + g.nw);
    if (lane == 0) { cv[g.wid] = bv; ci[g.wid] = bi; }
    g.sync();
    ++r;
  }
  for (int j = g.wid; j < r; j += g.nw) {
    double* p = A + (int64_t)ord[j] * lda;
    const double sc = scal[j];
    for (int e = j + 1 + lane; e < m; e += 32) p[e] *= sc;
    if (lane == 0) p[j] = beta[j];
  }
  g.sync();
  return r;
}

// Entry (i, c) of the kept rows R P^T of g_rrqr's factorization, in the
// original column order.
FRANK_D double rrqr_r(const double* A, int64_t lda, const int* at, int i, int c) {
  return at[c] >= i ? A[i + (int64_t)c * lda] : 0.0;
}

// X (m x r, ldx) = H_0 ... H_{k-1} X_0 for the first k reflectors of g_rrqr, X_0
// = [I; 0] (ident; k = r) or the k x r matrix X0 (ldx0, column perm[c] of it
// for column c where perm is given) on top of zeros.  A column belongs to
// eight lanes, its entries in registers (m <= 8 NR); reflectors beyond a unit
// column's own index leave it alone; no barrier before the end.
template <int NR>
FRANK_D void g_apply_cols(const Grp& g, int m, int k, int r, const double* A, int lda, const double* tau,
                          const int* ord, bool ident, const double* X0, int64_t ldx0, const int* perm, double* X,
                          int64_t ldx) {
  const int lane = threadIdx.x & 31, sub = lane >> 3, l8 = lane & 7, ng = 4 * g.nw;
  for (int c0 = 4 * g.wid; c0 < r; c0 += ng) {
    const int c = c0 + sub;
    const int top = ident ? min(k - 1, c0 + 3) : k - 1;
    double xr[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int e = l8 + 8 * i;
      xr[i] = ident ? (e == c ? 1.0 : 0.0) : (c < r && e < k ? X0[e + (int64_t)(perm ? perm[c] : c) * ldx0] : 0.0);
    }
    for (int j = top; j >= 0; --j) {
      const double* v = A + (int64_t)ord[j] * lda;
      const double t = tau[j];
      double vr[NR], d = 0.0;
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int e = l8 + 8 * i;
        vr[i] = (e > j && e < m) ? v[e] : (e == j ? 1.0 : 0.0);
        d = fma(vr[i], xr[i], d);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      d *= t;
#pragma unroll
      for (int i = 0; i < NR; ++i) xr[i] = fma(-d, vr[i], xr[i]);
    }
    if (c < r)
#pragma unroll
      for (int i = 0; i < NR; ++i)
        if (l8 + 8 * i < m) X[(l8 + 8 * i) + (int64_t)c * ldx] = xr[i];
  }
}

constexpr int G_COLS_MAX = 256;   // rows the register columns of g_apply_cols hold
static __device__ __noinline__ void g_apply_rrqr(Grp g, int m, int k, int r, const double* A, int lda, const double* tau,
                                          const int* ord, bool ident, const double* X0, int64_t ldx0,
                                          const int* perm, double* X, int64_t ldx) {
  if (m <= 48) g_apply_cols<6>(g, m, k, r, A, lda, tau, ord, ident, X0, ldx0, perm, X, ldx);
  else if (m <= 96) g_apply_cols<12>(g, m, k, r, A, lda, tau, ord, ident, X0, ldx0, perm, X, ldx);
  else g_apply_cols<G_COLS_MAX / 8>(g, m, k, r, A, lda, tau, ord, ident, X0, ldx0, perm, X, ldx);
  g.sync();
}

// Shared-memory leading dimension of a g_rrqr matrix: 8 mod 16, so that the
// lane groups of two columns read distinct banks.
FRANK_HD int rrqr_ld(int m) { return ((m + 7) & ~15) + 8; }

// Column-pivoted QR with randomized block pivoting (Martinsson, Quintana-Orti,
// Heavner, van de Geijn, "Householder QR factorization with randomization for
// column pivoting (HQRRP)", SIAM J. Sci. Comput. 39, 2017) of A (m x n, lda,
// global memory), for cores too large for shared memory: per panel of w
// columns a sketch Y = Omega A_trail (w + 8 rows, Omega uniform in [-1, 1)
// from a counter-based hash) picks the panel's pivots by g_rrqr in shared
// memory, the chosen columns move to the panel, and an unpivoted blocked step
// factors it and updates the rest by two products.  The stopping rule is the
// column-by-column one, evaluated exactly: after each panel the norms of every
// remaining column at every step t of the panel follow from the updated rows
// (later reflectors act orthogonally below row t), and the rank is the first
// step whose remaining columns are all at most thr.  On return A holds the
// clean V of each panel, Tf its T factors (panels of w), R (min(m, n) x n,
// ldr) the rows of R, jpvt[c] the original column at position c.  The pivots
// are a randomized choice, so ranks can differ from the column-by-column
// search by a few.  om: (w + 8) m doubles; region: shared, cap doubles;
// iscr: 3 GQ ints (shared); mx: GQ + 1 words (shared); nrm2: n doubles.
FRANK_D double sketch_omega(uint64_t k) {
  k += 0x9E3779B97F4A7C15ull;
  k = (k ^ (k >> 30)) * 0xBF58476D1CE4E5B9ull;
  k = (k ^ (k >> 27)) * 0x94D049BB133111EBull;
  k ^= k >> 31;
  return (double)(k >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// Panel width and shared memory (doubles) of g_rand_qrcp: the sketch with its
// vectors, or the panel, whichever is larger.
FRANK_HD int64_t rand_qrcp_smem(int m, int n, int w) {
  const int64_t sk = (int64_t)rrqr_ld(w + 8) * n + 8 * (w + 8) + 4 * 16 + n;
  const int64_t pn = (int64_t)panel_ld(m) * w;
  return sk > pn ? sk : pn;
}

static __device__ __noinline__ int g_rand_qrcp(Grp g, int m, int n, double* A, int64_t lda, double* R, int64_t ldr,
                                        double thr, int maxr, int w, int* jpvt, double* Tf, double* om, double* nrm2,
                                        double* region, int* iscr, unsigned long long* mx, GrpShared& s,
                                        GrpScratch x) {
  const int lane = threadIdx.x & 31;
  const int mind = min(min(m, n), maxr);
  for (int c = g.tid; c < n; c += g.nt) jpvt[c] = c;
  if (g.tid <= GQ) mx[g.tid] = 0ull;
  g.sync();
  // the first test: every column at most thr
  double best = 0.0;
  for (int c = g.wid; c < n; c += g.nw) {
    double s2 = 0.0;
    for (int e = lane; e < m; e += 32) s2 = fma(A[e + (int64_t)c * lda], A[e + (int64_t)c * lda], s2);
    best = fmax(best, warp_sum(s2));
  }
  if (lane == 0) atomicMax(mx, (unsigned long long)__double_as_longlong(best));
  g.sync();
  best = __longlong_as_double((long long)mx[0]);
  g.sync();
  if (mind == 0 || !(sqrt(best) > thr)) return 0;
  int r = 0;
  for (int panel = 0; r < mind; ++panel) {
    const int b = min(w, mind - r), mr = m - r, nr = n - r, sb = min(b + 8, mr);
    double* At = A + r + (int64_t)r * lda;
    for (int64_t e = g.tid; e < (int64_t)sb * mr; e += g.nt) om[e] = sketch_omega(((uint64_t)panel << 40) ^ (uint64_t)e);
    const int ldy = rrqr_ld(sb);
    double* Y = region;
    double* tau = Y + (int64_t)ldy * nr;
    double* vec = tau + sb;
    double* cand = vec + 2 * sb;
    int* ord = reinterpret_cast<int*>(cand + 4 * g.nw);
    int* at = ord + ((sb + 1) & ~1);
    g.sync();
    g_gemm(g, sb, nr, mr, 1.0, om, sb, false, At, lda, false, 0.0, Y, ldy, s.part);
    const int got = g_rrqr(g, sb, nr, Y, ldy, -1.0, b, tau, ord, at, vec, cand);
    if (got < b) return r;   // not a number in the sketch: no pivots to take
    // the chosen columns go to positions 0 .. b-1 in order; the columns they
    // displace go to the places they leave
    int *cho = iscr, *dsp = iscr + GQ, *vac = iscr + 2 * GQ;
    if (g.wid == 0) {
      const int c = lane < got ? ord[lane] : -1;
      const unsigned out = __ballot_sync(0xffffffffu, c >= b);
      const bool kept = lane < b && at[min(lane, nr - 1)] < got;   // position `lane` holds a chosen column
      const unsigned free_ = __ballot_sync(0xffffffffu, lane < b && !kept);
      const unsigned below = (1u << lane) - 1u;
      if (lane < b) cho[lane] = c;
      if (c >= b) vac[__popc(out & below)] = c;
      if (lane < b && !kept) dsp[__popc(free_ & below)] = lane;
      if (lane == 0) *reinterpret_cast<int*>(mx) = __popc(out);
    }
    g.sync();
    const int nd = *reinterpret_cast<int*>(mx);
    for (int e = g.tid; e <= m; e += g.nt) {
      if (e < m) {
        double* row = A + e + (int64_t)r * lda;
        double v[GQ];
#pragma unroll
        for (int t = 0; t < GQ; ++t)
          if (t < b) v[t] = row[(int64_t)cho[t] * lda];
        for (int t = 0; t < nd; ++t) row[(int64_t)vac[t] * lda] = row[(int64_t)dsp[t] * lda];
#pragma unroll
        for (int t = 0; t < GQ; ++t)
          if (t < b) row[(int64_t)t * lda] = v[t];
        // the finished rows of R above the panel move with their columns
        if (e < r) {
          double* rr = R + e + (int64_t)r * ldr;
#pragma unroll
          for (int t = 0; t < GQ; ++t)
            if (t < b) v[t] = rr[(int64_t)cho[t] * ldr];
          for (int t = 0; t < nd; ++t) rr[(int64_t)vac[t] * ldr] = rr[(int64_t)dsp[t] * ldr];
#pragma unroll
          for (int t = 0; t < GQ; ++t)
            if (t < b) rr[(int64_t)t * ldr] = v[t];
        }
      } else {
        int v[GQ];
#pragma unroll
        for (int t = 0; t < GQ; ++t)
          if (t < b) v[t] = jpvt[r + cho[t]];
        for (int t = 0; t < nd; ++t) jpvt[r + vac[t]] = jpvt[r + dsp[t]];
#pragma unroll
        for (int t = 0; t < GQ; ++t)
          if (t < b) jpvt[r + t] = v[t];
      }
    }
    g.sync();
    // one panel of b columns and its trailing update
    {
      const int ldp = panel_ld(mr);
      double* smP = region;
      double* Rp = R + r + (int64_t)r * ldr;
      for (int c = g.wid; c < b; c += g.nw)
#pragma unroll 4
        for (int e = lane; e < mr; e += 32) smP[e + c * ldp] = At[e + (int64_t)c * lda];
      for (int c = g.wid; c < b; c += g.nw)
        for (int e = r + b + lane; e < min(m, n); e += 32) R[e + (int64_t)(r + c) * ldr] = 0.0;
      g.sync();
      g_panel_qr(g, mr, b, smP, ldp, Rp, ldr, s);
      for (int c = g.wid; c < b; c += g.nw)
#pragma unroll 4
        for (int e = lane; e < mr; e += 32) At[e + (int64_t)c * lda] = smP[e + c * ldp];
      for (int e = g.tid; e < GQ * GQ; e += g.nt) Tf[(int64_t)panel * GQ * GQ + e] = s.T[e];
      const int nc = nr - b;
      if (nc > 0) {
        double* Ac = At + (int64_t)b * lda;
        g_gemm_tn(g, b, nc, mr, 1.0, smP, ldp, Ac, lda, x.W, GQ, x.part, s.part);
        g_gemm(g, b, nc, b, 1.0, s.T, GQ, true, x.W, GQ, false, 0.0, x.W2, GQ, s.part);
        g_gemm(g, mr, nc, b, -1.0, smP, ldp, false, x.W2, GQ, false, 1.0, Ac, lda, s.part);
      }
      if (g.tid <= GQ) mx[g.tid] = 0ull;
      // rows of R right of the panel, and the squared norms below it
      for (int c = r + b + g.wid; c < n; c += g.nw) {
        double s2 = 0.0;
        for (int e = r + b + lane; e < m; e += 32) s2 = fma(A[e + (int64_t)c * lda], A[e + (int64_t)c * lda], s2);
        s2 = warp_sum(s2);
        if (lane == 0) nrm2[c] = s2;
        for (int e = lane; e < b; e += 32) R[r + e + (int64_t)c * ldr] = A[r + e + (int64_t)c * lda];
      }
      g.sync();
    }
    // maxima over the remaining columns per step t, as the bits of
    // non-negative doubles (ordered like unsigned integers)
    for (int c0 = r + b; c0 < n; c0 += g.nt) {
      const int c = c0 + g.tid;
      const bool on = c < n;
      double s2 = on ? nrm2[c] : 0.0;
      for (int t = b; t >= 0; --t) {
        if (t < b && on) {
          const double a = R[r + t + (int64_t)c * ldr];
          s2 = fma(a, a, s2);
        }
        double v = s2;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) atomicMax(mx + t, (unsigned long long)__double_as_longlong(v));
      }
    }
    for (int j = g.tid; j < b; j += g.nt) {
      double s2 = 0.0;
      for (int t = j; t >= 0; --t) {
        const double a = R[r + t + (int64_t)(r + j) * ldr];
        s2 = fma(a, a, s2);
        atomicMax(mx + t, (unsigned long long)__double_as_longlong(s2));
      }
    }
    g.sync();
    int stop = -1;
    for (int t = 0; t <= b; ++t)
      if (sqrt(__longlong_as_double((long long)mx[t])) <= thr) { stop = t; break; }
    g.sync();
    if (stop >= 0) return r + stop;
    r += b;
  }
  return r;
}

// One-sided (Hestenes) Jacobi on the columns of G (m x n, ldg; angles from rows
// [0, m), rotations applied to rows [0, m_rot)): on return the columns are
// mutually orthogonal.  Round-robin (circle) pairs, a pair per eight lanes,
// one barrier per round.  Rotation as Demmel and Veselic, "Jacobi's method is
// more accurate than QR", SIAM J. Matrix Anal. Appl. 13, 1992.  flags: 2 ints
// (shared).  Returns the number of sweeps, or -1 at the sweep limit.
static __device__ __noinline__ int g_jacobi(Grp g, int m, int n, double* G, int64_t ldg, int max_sweeps, int* flags,
                                     int m_rot) {
  const int lane = threadIdx.x & 31, sub = lane >> 3, l8 = lane & 7;
  const int N2 = n + (n & 1);
  const double tol = (double)(m > 1 ? m : 1) * 2.220446049250313e-16;
  if (n < 2) { g.sync(); return 0; }
  if (g.tid < 2) flags[g.tid] = 0;
  g.sync();
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    int* flag = flags + (sweep & 1);
    for (int round = 0; round < N2 - 1; ++round) {
      for (int p0 = 4 * g.wid; p0 < N2 / 2; p0 += 4 * g.nw) {
        const int pr = p0 + sub;
        int p = 0, q = 0;
        bool on = pr < N2 / 2;
        if (pr == 0) { p = N2 - 1; q = round; }
        else if (on) {
          p = round + pr; if (p >= N2 - 1) p -= N2 - 1;
          q = round - pr; if (q < 0) q += N2 - 1;
        }
        if (p >= n || q >= n) on = false;
        if (p > q) { const int t = p; p = q; q = t; }
        if (!on) p = q = 0;
        double* gp = G + (int64_t)p * ldg;
        double* gq = G + (int64_t)q * ldg;
        double a = 0.0, b = 0.0, h = 0.0;
#pragma unroll 4
        for (int i = l8; i < m; i += 8) {
          const double x = gp[i], y = gq[i];
          a = fma(x, x, a); b = fma(y, y, b); h = fma(x, y, h);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
          h += __shfl_xor_sync(0xffffffffu, h, o);
        }
        if (!on || a == 0.0 || b == 0.0 || fabs(h) <= tol * sqrt(a) * sqrt(b)) continue;
        const double zeta = (b - a) / (2.0 * h);
        const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = rsqrt(1.0 + t * t), s = c * t;
#pragma unroll 4
        for (int i = l8; i < m_rot; i += 8) {
          const double x = gp[i], y = gq[i];
          gp[i] = c * x - s * y;
          gq[i] = s * x + c * y;
        }
        if (l8 == 0) *flag = 1;
      }
      g.sync();
    }
    const int rotated = *flag;
    if (!rotated) { g.sync(); return sweep + 1; }
    if (g.tid == 0) flags[(sweep + 1) & 1] = 0;
    g.sync();
  }
  return -1;
}

}  // namespace frank
