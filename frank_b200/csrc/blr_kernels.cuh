// Kernels of the BLR-LU factor-and-solve path (sm_100a).
//
// Storage (all column-major):
//   * dense block (i,j): bmax x bmax slot, ld = bmax, of which bs(i) x bs(j) used;
//   * low-rank block (i,j) = U S V: U (bmax x kcap, ld bmax), S (kcap x kcap,
//     ld kcap), Vt = V^T (bmax x kcap, ld bmax); rank r = rank[i*nb+j] columns used.
// T is the working precision (double for the plain FP64 path, float for the
// mixed path); every small factorization (leaf getrf, stacked-basis QR, core
// SVD) is computed in FP64.
#pragma once

#include "common.cuh"

#include <algorithm>

namespace frank {

template <typename T>
struct BlrView {
  int nb, bmax, kcap;
  const int* off;    // [nb+1] block offsets
  const int* dslot;  // [nb*nb] dense slot or -1
  const int* lslot;  // [nb*nb] low-rank slot or -1
  int* rank;         // [nb*nb] current ranks (low-rank blocks)
  T* D;
  T* U;
  T* S;
  T* Vt;
  FRANK_D int bs(int i) const { return off[i + 1] - off[i]; }
  FRANK_D bool is_lr(int i, int j) const { return lslot[i * nb + j] >= 0; }
  FRANK_D T* dense(int i, int j) const { return D + (int64_t)dslot[i * nb + j] * bmax * bmax; }
  FRANK_D T* u(int i, int j) const { return U + (int64_t)lslot[i * nb + j] * bmax * kcap; }
  FRANK_D T* s(int i, int j) const { return S + (int64_t)lslot[i * nb + j] * kcap * kcap; }
  FRANK_D T* vt(int i, int j) const { return Vt + (int64_t)lslot[i * nb + j] * bmax * kcap; }
};


// Per-factorization workspace (device pointers).
template <typename T>
struct FactorWs {
  int* perm;      // [nb][bmax]: row i of P*B is row perm[i] of B, per diagonal block
  int* ipiv;      // [nb][bmax]: LAPACK-style 0-based pivots per diagonal block
  T* Linv;        // [nb][bmax*bmax]: unit-lower inverse per diagonal block
  T* Uinv;        // [nb][bmax*bmax]: upper inverse per diagonal block
  T* UinvT;       // its transpose, or null where the caller keeps none
  T* WL;          // [nb][bmax*bmax]: (S V)^T of column-panel blocks, by block row
  T* WU;          // [nb][bmax*bmax]: U S of row-panel blocks, by block column
  double* getrf_scratch;  // leaf_scratch(bmax) doubles (k_getrf: bmax*bmax + 32*bmax)
  double* dscratch;       // dense-update scratch, per CTA slot
  int64_t dscratch_stride;
  double* rscratch;       // recompression scratch, per CTA slot
  int64_t rscratch_stride;
  int* err;
  int* work;                  // [nb] per-step work counters of the recompression
  unsigned long long* flops;  // [FLOP_SLOTS]
  int fixed_rank;
  double eps;
};

// Algorithmic FLOPs of one rounded LowRank addition as the reference issues it
// (gemm.cpp:253-272 then addition.cpp:93-127), counted with the LAWN 41
// operation counts: the inner product S_A V_A U_B S_B, U_C S_C and U_B S_B,
// geqrf + orgqr of Uc (m x s), gerqf + orgrq of VcT (s x n), the core gemm,
// dgesvd of the s x s core (22 s^3) and the two basis gemms.
FRANK_HD double rounded_addition_flops(double m, double n, double bi, double kc, double p, double q, double r) {
  const double s = fmin(kc + q, fmin(m, n));
  double f = 2.0 * p * p * bi + 2.0 * bi * q * q + 2.0 * p * bi * q;   // core of the product
  f += 2.0 * m * kc * kc + 2.0 * m * p * q;                               // U_C S_C, U_B S_B
  f += 4.0 * m * s * s - 4.0 / 3.0 * s * s * s;                           // geqrf + orgqr
  f += 4.0 * n * s * s - 4.0 / 3.0 * s * s * s;                           // gerqf + orgrq
  f += 2.0 * s * s * s + 22.0 * s * s * s;                                // Ru RvT, gesvd
  f += 2.0 * m * s * r + 2.0 * n * s * r;                                 // new U, V
  return f;
}

// Algorithmic FLOPs of one fast rounded addition (addition.cpp:133-189) as
// the reference issues it: projections Zu = U_C^T U_B, Zv, the residual bases,
// their QR / RQ with explicit factors, the (kc+p) x (kc+q) core, its SVD and
// the new bases [U_C | Q_u] U_m, V_m [V_C; Q_v].
FRANK_HD double fast_rounded_addition_flops(double m, double n, double bi, double kc, double p, double q, double r) {
  double f = 2.0 * p * p * bi + 2.0 * bi * q * q + 2.0 * p * bi * q;   // core of the product
  f += 4.0 * m * kc * p + 4.0 * n * kc * q;                               // Zu, Yu; Zv, Yv
  f += 4.0 * m * p * p - 4.0 / 3.0 * p * p * p;                           // geqrf + orgqr of Yu
  f += 4.0 * n * q * q - 4.0 / 3.0 * q * q * q;                           // gerqf + orgrq of Yv^T
  const double s = fmax(kc + p, kc + q);
  f += 4.0 * s * s * s + 22.0 * s * s * s;                                // core M, gesvd
  f += 2.0 * m * (kc + p) * r + 2.0 * n * (kc + q) * r;                   // new U, V
  return f;
}

// ---------------------------------------------------------------------------
// Reset the working copy from A_H (FP64) -- only the used parts are copied.
// One CTA per block.
// ---------------------------------------------------------------------------
template <typename T>
FRANK_D void k_reset_impl(BlrView<double> H, BlrView<T> W) {
  const int blk = blockIdx.x;
  const int i = blk / H.nb, j = blk % H.nb;
  const int bi = H.bs(i), bj = H.bs(j);
  if (H.lslot[blk] >= 0) {
    const int r = H.rank[blk];
    const double* hu = H.u(i, j); const double* hs = H.s(i, j); const double* hv = H.vt(i, j);
    T* wu = W.u(i, j); T* ws = W.s(i, j); T* wv = W.vt(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)bi * r; e += blockDim.x) {
      const int rr = e % bi, c = e / bi;
      wu[rr + (int64_t)c * W.bmax] = T(hu[rr + (int64_t)c * H.bmax]);
    }
    for (int64_t e = threadIdx.x; e < (int64_t)bj * r; e += blockDim.x) {
      const int rr = e % bj, c = e / bj;
      wv[rr + (int64_t)c * W.bmax] = T(hv[rr + (int64_t)c * H.bmax]);
    }
    for (int64_t e = threadIdx.x; e < (int64_t)r * r; e += blockDim.x) {
      const int rr = e % r, c = e / r;
      ws[rr + (int64_t)c * W.kcap] = T(hs[rr + (int64_t)c * H.kcap]);
    }
    if (threadIdx.x == 0) W.rank[blk] = r;
  } else if (H.dslot[blk] >= 0) {
    const double* hd = H.dense(i, j);
    T* wd = W.dense(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)bi * bj; e += blockDim.x) {
      const int rr = e % bi, c = e / bi;
      wd[rr + (int64_t)c * W.bmax] = T(hd[rr + (int64_t)c * H.bmax]);
    }
  }
}

template <typename T>
__global__ void k_reset(BlrView<double> H, BlrView<T> W) {
  k_reset_impl<T>(H, W);
}

// ---------------------------------------------------------------------------
// K0': truncation of the working copy's low-rank blocks to the factor
// tolerance (mixed plans, whose factor is computed at a looser tolerance
// than A_H).  Block U S V^T of A_H with orthonormal U, V: truncated pivoted
// QR of S to thr_scale * ||S||_F (the core truncation of the recompression,
// geqp3.cpp:71-192), S P = Q R, then RQ of the kept rows R P^T = S' Q', so
// W = (U Q_r) S' (V Q'^T)^T with rank r.  Blocks whose rank does not drop
// keep the copy k_reset made.  One CTA per block (grid-stride), FP64
// scratch slot per CTA (4 k^2 + 8 k doubles).
// ---------------------------------------------------------------------------
constexpr int TRUNC_THREADS = 256;

// Orthonormal bases for low-rank blocks given by the caller
// (frank_blr_set_lowrank): U = Qu Ru and V^T = Qv Rv by Householder QR, stored
// as U <- Qu, V^T <- Qv, S <- Ru S Rv^T -- the same matrix, with the
// orthonormal bases that the reset truncation and the projected additions
// assume (the on-device constructions produce them already).  One CTA per
// block at a time; scratch per CTA: 2 (bmax + kcap) kcap + 3 kcap^2 doubles.
constexpr int ORTH_THREADS = 256;
static __global__ void __launch_bounds__(ORTH_THREADS) k_orthonormalize_lr(BlrView<double> H, double* scratch,
                                                                   int64_t stride) {
  __shared__ double gsm[2 * 16 * 64];
  __shared__ double red[32];
  double* base = scratch + (int64_t)blockIdx.x * stride;
  const int nblk = H.nb * H.nb;
  for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
    if (H.lslot[blk] < 0) continue;
    const int k = H.rank[blk];
    const int i = blk / H.nb, j = blk % H.nb;
    const int bi = H.bs(i), bj = H.bs(j);
    if (k < 1 || k > bi || k > bj) continue;
    double* A1 = base;                        // bi x k, then its reflectors
    double* A2 = A1 + (int64_t)bi * k;        // bj x k
    double* Q = A2 + (int64_t)bj * k;         // max(bi, bj) x k
    double* Ru = Q + (int64_t)max(bi, bj) * k;
    double* Rv = Ru + (int64_t)k * k;
    double* Tmp = Rv + (int64_t)k * k;
    double* tu = Tmp + (int64_t)k * k;
    double* tv = tu + k;
    double* hu = H.u(i, j);
    double* hv = H.vt(i, j);
    double* hs = H.s(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)bi * k; e += blockDim.x) A1[e] = hu[(e % bi) + (e / bi) * H.bmax];
    for (int64_t e = threadIdx.x; e < (int64_t)bj * k; e += blockDim.x) A2[e] = hv[(e % bj) + (e / bj) * H.bmax];
    __syncthreads();
    cta_householder_qr(bi, k, A1, bi, tu, red);
    cta_householder_qr(bj, k, A2, bj, tv, red);
    for (int64_t e = threadIdx.x; e < (int64_t)k * k; e += blockDim.x) {
      const int r = e % k, c = e / k;
      Ru[e] = r <= c ? A1[r + (int64_t)c * bi] : 0.0;
      Rv[e] = r <= c ? A2[r + (int64_t)c * bj] : 0.0;
    }
    __syncthreads();
    // S <- Ru S Rv^T
    cta_gemm<double, ORTH_THREADS>(k, k, k, 1.0, Ru, k, false, hs, H.kcap, false, 0.0, Tmp, k, gsm);
    cta_gemm<double, ORTH_THREADS>(k, k, k, 1.0, Tmp, k, false, Rv, k, true, 0.0, hs, H.kcap, gsm);
    // U <- Qu, V^T <- Qv (explicit, from the reflectors)
    for (int side = 0; side < 2; ++side) {
      const int m = side ? bj : bi;
      const double* R = side ? A2 : A1;
      for (int64_t e = threadIdx.x; e < (int64_t)m * k; e += blockDim.x) Q[e] = ((e % m) == (e / m)) ? 1.0 : 0.0;
      __syncthreads();
      cta_apply_q(m, k, R, m, side ? tv : tu, k, Q, (int64_t)m);
      double* out = side ? hv : hu;
      for (int64_t e = threadIdx.x; e < (int64_t)m * k; e += blockDim.x) out[(e % m) + (e / m) * H.bmax] = Q[e];
      __syncthreads();
    }
  }
}

template <typename T>
FRANK_D void k_truncate_lr_impl(BlrView<double> H, BlrView<T> W, FactorWs<T> ws,
                                                              double thr_scale, double* scratch, int64_t stride) {
  __shared__ double gsm[2 * 16 * 64];
  __shared__ double red[32];
  __shared__ int redi[32];
  double* base = scratch + (int64_t)blockIdx.x * stride;
  const int nblk = H.nb * H.nb;
  for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
    if (H.lslot[blk] < 0) continue;
    const int k = H.rank[blk];
    if (k <= 1) continue;
    const int i = blk / H.nb, j = blk % H.nb;
    const int bi = H.bs(i), bj = H.bs(j);
    double* M = base;                          // k x k
    double* Xo = M + (int64_t)k * k;           // k x r
    double* X2 = Xo + (int64_t)k * k;          // k x r
    double* Qt = X2 + (int64_t)k * k;          // k x r
    double* tau = Qt + (int64_t)k * k;
    double* tau2 = tau + k;
    double* cn = tau2 + k;
    double* pn = cn + k;
    int* jpvt = reinterpret_cast<int*>(pn + k);
    int* jinv = jpvt + k;
    const double* hs = H.s(i, j);
    double f = 0.0;
    for (int e = threadIdx.x; e < k * k; e += blockDim.x) {
      const double v = hs[(e % k) + (int64_t)(e / k) * H.kcap];
      M[e] = v;
      f += v * v;
    }
    f = block_sum(f, red);
    const int r = cta_truncated_geqp3(k, k, M, k, thr_scale * sqrt(f), W.kcap, tau, cn, pn, jpvt, red, redi);
    if (r >= k) continue;
    T* wu = W.u(i, j); T* wsm = W.s(i, j); T* wv = W.vt(i, j);
    if (r == 0) {
      for (int e = threadIdx.x; e < bi; e += blockDim.x) wu[e] = T(e == 0 ? 1.0 : 0.0);
      for (int e = threadIdx.x; e < bj; e += blockDim.x) wv[e] = T(e == 0 ? 1.0 : 0.0);
      if (threadIdx.x == 0) { wsm[0] = T(0); W.rank[blk] = 1; }
      __syncthreads();
      continue;
    }
    // Xo = Q[:, :r]
    for (int e = threadIdx.x; e < k * r; e += blockDim.x) Xo[e] = ((e % k) == (e / k)) ? 1.0 : 0.0;
    for (int c = threadIdx.x; c < k; c += blockDim.x) jinv[jpvt[c]] = c;
    __syncthreads();
    cta_apply_q(k, r, M, k, tau, r, Xo, (int64_t)k);
    // RQ of R P^T (r x k): QR of X2 = (R P^T)^T J
    for (int e = threadIdx.x; e < k * r; e += blockDim.x) {
      const int c = e % k, a = e / k;
      const int row = r - 1 - a, src = jinv[c];
      X2[e] = (row <= src) ? M[row + (int64_t)src * k] : 0.0;
    }
    __syncthreads();
    cta_householder_qr(k, r, X2, k, tau2, red);
    for (int e = threadIdx.x; e < r * r; e += blockDim.x) {
      const int a = e % r, c = e / r;
      const int ra = r - 1 - c, ca = r - 1 - a;
      wsm[a + (int64_t)c * W.kcap] = T((ra <= ca) ? X2[ra + (int64_t)ca * k] : 0.0);
    }
    for (int e = threadIdx.x; e < k * r; e += blockDim.x) Qt[e] = ((e % k) == (e / k)) ? 1.0 : 0.0;
    __syncthreads();
    cta_apply_q(k, r, X2, k, tau2, r, Qt, (int64_t)k);
    // new U = U Xo; then Xo := Qt with its columns reversed, new V = V Xo
    cta_gemm<double, TRUNC_THREADS>(bi, r, k, 1.0, H.u(i, j), H.bmax, false, Xo, k, false, 0.0, wu, W.bmax, gsm);
    for (int e = threadIdx.x; e < k * r; e += blockDim.x) {
      const int rr = e % k, a = e / k;
      Xo[e] = Qt[rr + (int64_t)(r - 1 - a) * k];
    }
    __syncthreads();
    cta_gemm<double, TRUNC_THREADS>(bj, r, k, 1.0, H.vt(i, j), H.bmax, false, Xo, k, false, 0.0, wv, W.bmax, gsm);
    if (threadIdx.x == 0) W.rank[blk] = r;
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(TRUNC_THREADS) k_truncate_lr(BlrView<double> H, BlrView<T> W, FactorWs<T> ws,
                                                              double thr_scale, double* scratch, int64_t stride) {
  k_truncate_lr_impl<T>(H, W, ws, thr_scale, scratch, stride);
}

// ---------------------------------------------------------------------------
// Dense getrf with partial pivoting, FP64, one CTA (512 threads), for the entry
// point that may not allocate (plans factor their leaves by column tiles on
// several CTAs, k_leaf_step).  Blocked right-looking LU (panel width 32): the panel is
// factored column by column (idamax pivot, row swap across the whole block,
// reciprocal scaling and rank-1 update as in LAPACK dgetf2), then the row
// block is solved with the unit-lower 32x32 triangle and the trailing matrix
// updated by a CTA GEMM.  Writes the packed LU back into the block and the
// pivots/permutation.
// ---------------------------------------------------------------------------
constexpr int GETRF_THREADS = 512;

// One 32-column panel step of the leaf LU of a b x b FP64 matrix Wm (ld b):
// partial-pivoted factorization of columns jb .. jb+jn-1 (in registers, one
// row per thread, when b <= GETRF_THREADS; column steps on the global copy
// otherwise), the panel's interchanges applied to every other column, and
// U12 = L11^{-1} A12 (through the 32 x bmax scratch panel Gp).  Pivots into
// piv[jb ..]; returns the first column with a zero pivot, or -1.  Called by
// all threads of a GETRF_THREADS CTA.
FRANK_D int getrf_panel_step(int b, int jb, double* Wm, double* Gp, int* piv, double* red, int* redi, double* gsm,
                             double* tri, double* prow, double* xrow) {
  const int jn = min(32, b - jb);
  int zero = -1;
  if (b <= GETRF_THREADS) {
    // Panel in registers: thread t owns row t (t >= jb) and its jn panel
    // entries; a column step is an arg-max, a row exchange through shared
    // memory and a rank-1 update, with no global traffic.
    const int t = threadIdx.x;
    const bool own = (t >= jb && t < b);
    double a[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) a[c] = (own && c < jn) ? Wm[t + (int64_t)(jb + c) * b] : 0.0;
    for (int jj = 0; jj < jn; ++jj) {
      const int j = jb + jj;
      double v = -1.0;
      int vi = -1;
      if (t >= j && t < b) {
#pragma unroll
        for (int c = 0; c < 32; ++c) if (c == jj) v = fabs(a[c]);
        vi = t;
      }
      double amax;
      const int p = block_argmax_abs(v < 0.0 ? 0.0 : v, vi, red, redi, &amax);
      if (threadIdx.x == 0) piv[j] = p;
      if (amax == 0.0 && zero < 0) zero = j;
      // the pivot row goes to row j, row j to row p
      if (t == p) {
#pragma unroll
        for (int c = 0; c < 32; ++c) prow[c] = a[c];
      }
      if (t == j) {
#pragma unroll
        for (int c = 0; c < 32; ++c) xrow[c] = a[c];
      }
      __syncthreads();
      if (t == j) {
#pragma unroll
        for (int c = 0; c < 32; ++c) a[c] = prow[c];
      } else if (t == p) {
#pragma unroll
        for (int c = 0; c < 32; ++c) a[c] = xrow[c];
      }
      if (t > j && t < b && amax != 0.0) {
        const double rcp = 1.0 / prow[jj];
        double l = 0.0;
#pragma unroll
        for (int c = 0; c < 32; ++c) if (c == jj) { a[c] *= rcp; l = a[c]; }
#pragma unroll
        for (int c = 0; c < 32; ++c) if (c > jj) a[c] -= l * prow[c];
      }
      __syncthreads();
    }
    if (own) {
#pragma unroll
      for (int c = 0; c < 32; ++c) if (c < jn) Wm[t + (int64_t)(jb + c) * b] = a[c];
    }
    __syncthreads();
    // the panel's interchanges applied to the columns outside the panel
    for (int c = threadIdx.x; c < b; c += blockDim.x) {
      if (c >= jb && c < jb + jn) continue;
      double* col = Wm + (int64_t)c * b;
      for (int jj = 0; jj < jn; ++jj) {
        const int j = jb + jj, p = piv[j];
        if (p != j) { const double tmp = col[j]; col[j] = col[p]; col[p] = tmp; }
      }
    }
    __syncthreads();
  } else {
    // blocks larger than the thread count: column steps on the global copy
    for (int j = jb; j < jb + jn; ++j) {
      double best = -1.0;
      int bi = -1;
      for (int r = j + threadIdx.x; r < b; r += blockDim.x) {
        const double av = fabs(Wm[r + (int64_t)j * b]);
        if (av > best) { best = av; bi = r; }
      }
      double amax;
      const int p = block_argmax_abs(best < 0.0 ? 0.0 : best, bi, red, redi, &amax);
      if (threadIdx.x == 0) piv[j] = p;
      if (amax == 0.0 && zero < 0) zero = j;
      if (p != j && amax != 0.0) {
        for (int c = threadIdx.x; c < b; c += blockDim.x) {
          const double tt = Wm[j + (int64_t)c * b];
          Wm[j + (int64_t)c * b] = Wm[p + (int64_t)c * b];
          Wm[p + (int64_t)c * b] = tt;
        }
      }
      __syncthreads();
      if (amax != 0.0) {
        const double rcp = 1.0 / Wm[j + (int64_t)j * b];
        for (int r = j + 1 + threadIdx.x; r < b; r += blockDim.x) Wm[r + (int64_t)j * b] *= rcp;
      }
      __syncthreads();
      const int nr = b - j - 1, nc = jb + jn - j - 1;
      for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
        const int r = j + 1 + e % nr, c = j + 1 + e / nr;
        Wm[r + (int64_t)c * b] -= Wm[r + (int64_t)j * b] * Wm[j + (int64_t)c * b];
      }
      __syncthreads();
    }
  }
  // U12 = L11^{-1} A12: invert the unit-lower 32x32 L11 into tri, then a
  // CTA GEMM into the scratch panel and back.
  const int ncr = b - jb - jn;
  if (ncr > 0) {
    for (int e = threadIdx.x; e < 32 * 33; e += blockDim.x) tri[e] = 0.0;
    __syncthreads();
    if (threadIdx.x < jn) {
      const int c = threadIdx.x;
      tri[c + c * 33] = 1.0;
      for (int r = c + 1; r < jn; ++r) {
        double s = 0.0;
        for (int t = c; t < r; ++t) s += Wm[(jb + r) + (int64_t)(jb + t) * b] * tri[t + c * 33];
        tri[r + c * 33] = -s;
      }
    }
    __syncthreads();
    cta_gemm<double, GETRF_THREADS>(jn, ncr, jn, 1.0, tri, 33, false, Wm + jb + (int64_t)(jb + jn) * b, b, false,
                                    0.0, Gp, 32, gsm);
    for (int e = threadIdx.x; e < jn * ncr; e += blockDim.x) {
      const int r = e % jn, c = e / jn;
      Wm[(jb + r) + (int64_t)(jb + jn + c) * b] = Gp[r + (int64_t)c * 32];
    }
    __syncthreads();
  }
  return zero;
}

template <typename T>
__global__ void __launch_bounds__(GETRF_THREADS) k_getrf(BlrView<T> A, FactorWs<T> ws, int i) {
  __shared__ double red[32];
  __shared__ int redi[32];
  __shared__ double gsm[2 * 16 * 64];
  __shared__ double tri[32 * 33];
  const int b = A.bs(i);
  const int ldA = A.bmax;
  T* Dp = A.dense(i, i);
  double* Wm = ws.getrf_scratch;                       // b x b working matrix
  double* Gp = Wm + (int64_t)A.bmax * A.bmax;          // 32 x bmax product panel
  int* piv = ws.ipiv + (int64_t)i * A.bmax;
  int* perm = ws.perm + (int64_t)i * A.bmax;
  T* Li = ws.Linv + (int64_t)i * A.bmax * A.bmax;
  T* Ui = ws.Uinv + (int64_t)i * A.bmax * A.bmax;
  for (int64_t e = threadIdx.x; e < (int64_t)b * b; e += blockDim.x) {
    const int r = e % b, c = e / b;
    Wm[r + (int64_t)c * b] = double(Dp[r + (int64_t)c * ldA]);
  }
  __syncthreads();
  int first_zero = -1;
  __shared__ double prow[32];          // pivot row of the panel, broadcast
  __shared__ double xrow[32];          // row exchanged with the pivot row
  for (int jb = 0; jb < b; jb += 32) {
    const int jn = min(32, b - jb);
    {
      const int z = getrf_panel_step(b, jb, Wm, Gp, piv, red, redi, gsm, tri, prow, xrow);
      if (z >= 0 && first_zero < 0) first_zero = z;
    }
    const int m2 = b - jb - jn;
    if (m2 > 0)
      cta_gemm<double, GETRF_THREADS>(m2, m2, jn, -1.0, Wm + (jb + jn) + (int64_t)jb * b, b, false,
                                      Wm + jb + (int64_t)(jb + jn) * b, b, false, 1.0,
                                      Wm + (jb + jn) + (int64_t)(jb + jn) * b, b, gsm);
  }
  if (threadIdx.x == 0) {
    atomicAdd(ws.flops + FLOP_GETRF, (unsigned long long)(2.0 / 3.0 * (double)b * b * b));
    if (first_zero >= 0) atomicCAS(ws.err + ERR_SINGULAR_STEP, 0, i + 1);
    // permutation from the interchanges: (P B)[r] = B[perm[r]]
    for (int r = 0; r < b; ++r) perm[r] = r;
    for (int r = 0; r < b; ++r) {
      const int p = piv[r];
      const int t = perm[r]; perm[r] = perm[p]; perm[p] = t;
    }
  }
  // packed LU back into the block
  for (int64_t e = threadIdx.x; e < (int64_t)b * b; e += blockDim.x) {
    const int r = e % b, c = e / b;
    Dp[r + (int64_t)c * ldA] = T(Wm[r + (int64_t)c * b]);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// K1 as separate launches (the factorization path): the leaf LU of a b x b
// diagonal block by column tiles of W, one CTA per tile and one launch per
// panel.  Launch p: the CTA of tile p brings its tile up to date with panel
// p - 1 (row interchanges by a gather, U12 by substitution, the trailing
// product on the FP64 tensor pipe) and factors it as panel p, while the CTAs
// of the later tiles do the same update; the CTA of tile p - 1 inverts that
// panel's two W x W triangles for the explicit inverses below; earlier tiles
// apply the interchanges if there were any.  The tile lives in shared memory,
// the panel in registers (RPT rows of W entries per thread), rows are never
// moved: each thread keeps the position its row has been exchanged to.  A
// column step is one block barrier: each warp's pivot candidate (found on the
// integer halves of |a|, ties broken toward the smallest position as in
// idamax) goes to shared memory together with its row, eight columns wide;
// every eight columns the rest of the panel is updated at once.  A chain of b
// column steps bounds the whole thing, so what counts is the latency of a
// step (some 1100 cycles; an 8-panel leaf of b = 256 takes 270 us, its
// inverses included).  The scheme before (one CTA with six barriers per step,
// a serial triangle inverse and exchanges through L2, a second launch for the
// trailing tiles) took 96 us + 19 us per panel at b = 256 and 118 us + 21 us
// at b = 512.
// After the last panel, k_leaf_final stores the packed LU (tile CTAs) and
// forms Linv and Uinv: one CTA per column block of W of each, the block of
// the inverse in shared memory, right-looking over the row blocks -- multiply
// by the inverted diagonal triangle, then one product updates every row
// still to come -- so each of the b / W steps is two short products instead
// of one long inner-product chain (320 us at b = 256, 870 us at b = 512
// before).
// ---------------------------------------------------------------------------
constexpr int LEAF_THREADS = 512;
constexpr int LEAF_W = 32;            // panel width (b <= LEAF_THREADS)
constexpr int LEAF_W_WIDE = 16;       // panel width of larger blocks (two rows per thread)
constexpr int LEAF_WIDE_MAX = 1024;   // largest block order

FRANK_HD int leaf_width(int b) { return b <= LEAF_THREADS ? LEAF_W : LEAF_W_WIDE; }
// leading dimension of a tile in shared memory: 4 mod 16, so that the mma
// fragments (4 rows of 4 columns per phase) fall into distinct banks
FRANK_HD int leaf_lds(int b) { return ((b + 15) & ~15) + 4; }
inline int leaf_threads(int b) { return b <= LEAF_THREADS ? std::max(128, (b + 31) & ~31) : LEAF_THREADS; }
inline size_t leaf_smem(int b) { return (size_t)leaf_lds(b) * leaf_width(b) * sizeof(double); }
constexpr int LEAF_SMEM_MAX = (LEAF_THREADS + 4) * LEAF_W * (int)sizeof(double);
static_assert((LEAF_WIDE_MAX + 4) * LEAF_W_WIDE <= (LEAF_THREADS + 4) * LEAF_W, "tile sizes");
// doubles of FactorWs::getrf_scratch: the working matrix, the inverted
// diagonal triangles, the row maps of two panels and the exchange flags
inline int64_t leaf_scratch(int bmax) { return (int64_t)bmax * bmax + 66 * (int64_t)bmax + 4096; }

struct LeafScratch {
  double* Wm;     // b x b (ld b)
  double* dinv;   // per panel: Linv (W x W, ld W), Uinv
  int* src;       // [2][bmax]: row at position r before the panel's exchanges
  int* moved;     // [panels]: whether the panel exchanged any rows
};

template <int W>
FRANK_D LeafScratch leaf_view(double* base, int bmax) {
  LeafScratch s;
  const int npmax = (bmax + W - 1) / W;
  s.Wm = base;
  s.dinv = base + (int64_t)bmax * bmax;
  s.src = reinterpret_cast<int*>(s.dinv + (int64_t)npmax * 2 * W * W);
  s.moved = s.src + 2 * bmax;
  return s;
}

constexpr int LEAF_S = 8;             // columns between two updates of the rest of a panel

struct LeafShared {
  double tri[LEAF_W * (LEAF_W + 1)];
  alignas(16) double u[LEAF_W][LEAF_W + 2];          // rows of U of the panel
  double l11[LEAF_S][LEAF_S];                        // the sub-panel's triangle
  double2 crow[2][LEAF_THREADS / 32][LEAF_S / 2];    // each warp's candidate row
  uint4 cand[2][LEAF_THREADS / 32];
};

// Largest |a| among the lanes' candidates with ties toward the smallest
// position, as (high word, low word, position) in every lane: the bits of
// non-negative doubles are ordered like unsigned integers, so three integer
// warp reductions replace ten 64-bit shuffles.  pos = ~0u: no candidate.
FRANK_D uint4 warp_pivot(unsigned hi, unsigned lo, unsigned pos) {
  const bool on = pos != ~0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, on ? hi : 0u);
  const unsigned ml = __reduce_max_sync(0xffffffffu, on && hi == mh ? lo : 0u);
  const unsigned mp = __reduce_min_sync(0xffffffffu, on && hi == mh && lo == ml ? pos : ~0u);
  return make_uint4(mh, ml, mp, 0u);
}

// Columns j0 .. j0+7 of a panel whose current column is a[.][0] and whose NV
// first entries are live (the entries of the sub-panel shift down by one per
// step), then the update of its remaining NV - 8 columns at once.
template <int W, int RPT, int NV>
FRANK_D void leaf_columns(int m, int j0, int jn, double (&a)[RPT][W], unsigned (&pos)[RPT], unsigned& done, double* sm,
                          int lds, int* piv, int jb, int& zero, LeafShared& sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (j0 >= jn) return;
  const int j1 = min(jn, j0 + LEAF_S);
  for (int jj = j0; jj < j1; ++jj) {
    const int par = jj & 1;
    unsigned bh = 0u, bl = 0u, bp = ~0u;
    int bk = 0;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int row = threadIdx.x + k * blockDim.x;
      if (row < m && !((done >> k) & 1u)) {
        const double v = fabs(a[k][0]);
        const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
        if (bp == ~0u || h > bh || (h == bh && (l > bl || (l == bl && pos[k] < bp)))) { bh = h; bl = l; bp = pos[k]; bk = k; }
      }
    }
    const uint4 wc = warp_pivot(bh, bl, bp);
    // the warp's candidate with its row, so that the winner needs no second barrier
    if (bp != ~0u ? bp == wc.z : (wc.z == ~0u && lane == 0)) {
      sh.cand[par][wid] = wc;
#pragma unroll
      for (int x = 0; x < LEAF_S / 2; ++x) {
        double2 v = make_double2(a[0][2 * x], a[0][2 * x + 1]);
#pragma unroll
        for (int k = 1; k < RPT; ++k)
          if (bk == k) v = make_double2(a[k][2 * x], a[k][2 * x + 1]);
        sh.crow[par][wid][x] = v;
      }
    }
    __syncthreads();
    const uint4 q = lane < nw ? sh.cand[par][lane] : make_uint4(0u, 0u, ~0u, 0u);
    const uint4 c = warp_pivot(q.x, q.y, q.z);
    const int ww = __ffs(__ballot_sync(0xffffffffu, q.z == c.z)) - 1;
    const unsigned p = c.z;
    const bool nonzero = (c.x | c.y) != 0u;
    const double ra = 1.0 / __hiloint2double((int)c.x, (int)c.y);   // 1 / |pivot|
    double pr[LEAF_S];
#pragma unroll
    for (int x = 0; x < LEAF_S / 2; ++x) {
      const double2 v = sh.crow[par][ww][x];
      pr[2 * x] = v.x;
      pr[2 * x + 1] = v.y;
    }
    const double rcp = pr[0] < 0.0 ? -ra : ra;
    if (threadIdx.x == 0) {
      piv[jj] = jb + (int)p;
      if (!nonzero && zero < 0) zero = jb + jj;
#pragma unroll
      for (int x = 0; x < LEAF_S; ++x)
        if (jj + x < j0 + LEAF_S) sh.u[jj][jj + x] = pr[x];
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int row = threadIdx.x + k * blockDim.x;
      if (row < m && !((done >> k) & 1u)) {
        if (pos[k] == p) { pos[k] = jj; done |= 1u << k; }
        else if (pos[k] == (unsigned)jj) pos[k] = p;
      }
      const double l = nonzero ? a[k][0] * rcp : a[k][0];
      if (row < m && !((done >> k) & 1u)) sm[row + jj * lds] = l;
      const double lu = nonzero ? l : 0.0;
#pragma unroll
      for (int x = 1; x < LEAF_S; ++x) a[k][x - 1] = fma(-lu, pr[x], a[k][x]);
      a[k][LEAF_S - 1] = 0.0;
    }
  }
  if (NV <= LEAF_S || j0 + LEAF_S >= jn) return;
  // U12 = L11^{-1} A12 of the sub-panel's pivot rows, a column per lane
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int row = threadIdx.x + k * blockDim.x, i = (int)pos[k] - j0;
    if (row < m && ((done >> k) & 1u) && i >= 0 && i < LEAF_S) {
#pragma unroll
      for (int x = LEAF_S; x < NV; ++x) sh.u[j0 + i][j0 + x] = a[k][x];
      for (int t = 0; t < i; ++t) sh.l11[i][t] = sm[row + (j0 + t) * lds];
    }
  }
  __syncthreads();
  if (wid == 0 && lane < NV - LEAF_S) {
    double v[LEAF_S];
#pragma unroll
    for (int i = 0; i < LEAF_S; ++i) v[i] = sh.u[j0 + i][j0 + LEAF_S + lane];
#pragma unroll
    for (int t = 0; t < LEAF_S; ++t)
#pragma unroll
      for (int i = t + 1; i < LEAF_S; ++i) v[i] = fma(-sh.l11[i][t], v[t], v[i]);
#pragma unroll
    for (int i = 1; i < LEAF_S; ++i) sh.u[j0 + i][j0 + LEAF_S + lane] = v[i];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int row = threadIdx.x + k * blockDim.x;
    double l[LEAF_S];
#pragma unroll
    for (int t = 0; t < LEAF_S; ++t) l[t] = row < m && !((done >> k) & 1u) ? sm[row + (j0 + t) * lds] : 0.0;
#pragma unroll
    for (int x = LEAF_S; x < NV; x += 2) {
      double v = a[k][x], w = a[k][x + 1];
#pragma unroll
      for (int t = 0; t < LEAF_S; ++t) {
        const double2 u = *reinterpret_cast<const double2*>(&sh.u[j0 + t][j0 + x]);
        v = fma(-l[t], u.x, v);
        w = fma(-l[t], u.y, w);
      }
      a[k][x - LEAF_S] = v;
      a[k][x + 1 - LEAF_S] = w;
    }
  }
}

// Partial-pivoted LU of the panel in sm (m x jn, ld lds; rows jb .. b-1 of the
// block, columns jb ..), written to Wm in pivoted order with its pivots, row
// map, exchange flag and the running permutation perm.
template <int W, int RPT>
FRANK_D void leaf_panel(int b, int jb, double* sm, int lds, const LeafScratch& L, int par, int panel, int* piv,
                        int* perm, int* err, int step, LeafShared& sh) {
  const int m = b - jb, jn = min(W, m);
  double a[RPT][W];
  unsigned pos[RPT], done = 0u;
  int zero = -1;
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int row = threadIdx.x + k * blockDim.x;
    pos[k] = row;
#pragma unroll
    for (int c = 0; c < W; ++c) a[k][c] = (row < m && c < jn) ? sm[row + c * lds] : 0.0;
  }
  leaf_columns<W, RPT, W>(m, 0, jn, a, pos, done, sm, lds, piv + jb, jb, zero, sh);
  leaf_columns<W, RPT, W - 8>(m, 8, jn, a, pos, done, sm, lds, piv + jb, jb, zero, sh);
  if constexpr (W > 16) {
    leaf_columns<W, RPT, 16>(m, 16, jn, a, pos, done, sm, lds, piv + jb, jb, zero, sh);
    leaf_columns<W, RPT, 8>(m, 24, jn, a, pos, done, sm, lds, piv + jb, jb, zero, sh);
  }
  __syncthreads();
  if (threadIdx.x == 0 && zero >= 0) atomicCAS(err + ERR_SINGULAR_STEP, 0, step + 1);
  int mv = 0, pv[RPT];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int row = threadIdx.x + k * blockDim.x;
    pv[k] = 0;
    if (row >= m) continue;
    const int to = jb + (int)pos[k];
    const int pr = (int)pos[k];
    for (int c = 0; c < jn; ++c) L.Wm[to + (int64_t)(jb + c) * b] = pr < jn && c >= pr ? sh.u[pr][c] : sm[row + c * lds];
    L.src[par * b + to] = jb + row;
    pv[k] = jb == 0 ? row : perm[jb + row];
    mv |= (int)pos[k] != row;
  }
  mv = __syncthreads_or(mv);
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int row = threadIdx.x + k * blockDim.x;
    if (row < m) perm[jb + pos[k]] = pv[k];
  }
  if (threadIdx.x == 0) L.moved[panel] = mv;
}

// Inverses of the two W x W triangles of a factored panel (identity beyond
// the block): a warp per triangle, a column per lane in registers, the
// triangle's entries broadcast from shared memory.
template <int W>
FRANK_D void leaf_dinv(int b, int jb, const double* Wm, double* out, LeafShared& sh) {
  const int jn = min(W, b - jb);
  for (int e = threadIdx.x; e < W * W; e += blockDim.x) {
    const int r = e % W, c = e / W;
    sh.tri[r + c * (W + 1)] = (r < jn && c < jn) ? Wm[(jb + r) + (int64_t)(jb + c) * b] : (r == c ? 1.0 : 0.0);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid < 2) {
    double v[W];
#pragma unroll
    for (int r = 0; r < W; ++r) v[r] = r == lane ? 1.0 : 0.0;
    if (wid == 0) {
#pragma unroll
      for (int t = 0; t < W; ++t)
#pragma unroll
        for (int r = t + 1; r < W; ++r) v[r] = fma(-sh.tri[r + t * (W + 1)], v[t], v[r]);
    } else {
      const double rd = 1.0 / sh.tri[min(lane, W - 1) * (W + 2)];
#pragma unroll
      for (int t = W - 1; t >= 0; --t) {
        v[t] *= __shfl_sync(0xffffffffu, rd, t);
#pragma unroll
        for (int r = 0; r < t; ++r) v[r] = fma(-sh.tri[r + t * (W + 1)], v[t], v[r]);
      }
    }
    if (lane < W)
#pragma unroll
      for (int r = 0; r < W; ++r) out[(wid ? W * W : 0) + r + lane * W] = v[r];
  }
  __syncthreads();
}

template <typename T, int W, int RPT>
FRANK_D void leaf_step_body(const BlrView<T>& A, const FactorWs<T>& ws, int i, int p) {
  extern __shared__ double lsm[];
  __shared__ LeafShared sh;
  const int b = A.bs(i), ld = A.bmax, np = (b + W - 1) / W, q = blockIdx.x;
  if (p >= np || q >= np) return;
  const LeafScratch L = leaf_view<W>(ws.getrf_scratch, A.bmax);
  const int lds = leaf_lds(b);
  const int c0 = q * W, cn = min(W, b - c0);
  int* piv = ws.ipiv + (int64_t)i * ld;
  int* perm = ws.perm + (int64_t)i * ld;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* panel = lsm;
  if (p == 0) {
    const T* Dp = A.dense(i, i) + (int64_t)c0 * ld;
    for (int c = wid; c < cn; c += nw) {
#pragma unroll 4
      for (int r = lane; r < b; r += 32) {
        const double v = double(Dp[r + (int64_t)c * ld]);
        if (q == 0) lsm[r + c * lds] = v;
        else L.Wm[r + (int64_t)(c0 + c) * b] = v;
      }
    }
    if (q != 0) return;
    __syncthreads();
  } else {
    const int j0 = (p - 1) * W, m = b - j0, par = (p - 1) & 1;
    const int* src = L.src + par * b;
    if (q == p - 1) {
      leaf_dinv<W>(b, j0, L.Wm, L.dinv + (int64_t)q * 2 * W * W, sh);
      return;
    }
    const bool mv = L.moved[p - 1] != 0;
    if (q < p - 1 && !mv) return;
    // rows j0 .. b-1 of the tile, exchanged by panel p - 1
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
      const double* w = L.Wm + (mv ? src[j0 + r] : j0 + r) + (int64_t)c0 * b;
#pragma unroll 8
      for (int c = 0; c < cn; ++c) lsm[r + c * lds] = w[(int64_t)c * b];
    }
    if (q < p - 1) {
      __syncthreads();
      for (int r = threadIdx.x; r < m; r += blockDim.x)
        for (int c = 0; c < cn; ++c) L.Wm[(j0 + r) + (int64_t)(c0 + c) * b] = lsm[r + c * lds];
      return;
    }
    for (int e = threadIdx.x; e < W * W; e += blockDim.x)
      sh.tri[e % W + (e / W) * (W + 1)] = L.Wm[(j0 + e % W) + (int64_t)(j0 + e / W) * b];
    __syncthreads();
    // U12 = L11^{-1} A12 (panel p - 1 has W columns: only the last one can have fewer)
    // -- a column per lane, in registers
    if (wid == 0 && lane < cn) {
      double v[W];
#pragma unroll
      for (int r = 0; r < W; ++r) v[r] = lsm[r + lane * lds];
#pragma unroll
      for (int t = 0; t < W - 1; ++t)
#pragma unroll
        for (int r = t + 1; r < W; ++r) v[r] = fma(-sh.tri[r + t * (W + 1)], v[t], v[r]);
#pragma unroll
      for (int r = 0; r < W; ++r) lsm[r + lane * lds] = v[r];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < W * cn; e += blockDim.x)
      L.Wm[(j0 + e % W) + (int64_t)(c0 + e / W) * b] = lsm[e % W + (e / W) * lds];
    // trailing rows: -= L21 U12
    warps_dgemm<4, 2>(wid, nw, m - W, cn, W, -1.0, L.Wm + (j0 + W) + (int64_t)j0 * b, 1, b, lsm, lds, 1, 1.0, lsm + W,
                      lds);
    __syncthreads();
    if (q > p) {
      for (int c = wid; c < cn; c += nw)
        for (int r = W + lane; r < m; r += 32) L.Wm[(j0 + r) + (int64_t)(c0 + c) * b] = lsm[r + c * lds];
      return;
    }
    panel = lsm + W;
  }
  leaf_panel<W, RPT>(b, p * W, panel, lds, L, p & 1, p, piv, perm, ws.err, i, sh);
  if (p == np - 1) {
    __syncthreads();
    leaf_dinv<W>(b, p * W, L.Wm, L.dinv + (int64_t)p * 2 * W * W, sh);
  }
}

template <typename T>
FRANK_D void k_leaf_step_impl(const BlrView<T>& A, const FactorWs<T>& ws, int i, int p) {
  if (A.bmax <= LEAF_THREADS) leaf_step_body<T, LEAF_W, 1>(A, ws, i, p);
  else leaf_step_body<T, LEAF_W_WIDE, 2>(A, ws, i, p);
}

template <typename T>
__global__ void __launch_bounds__(LEAF_THREADS) k_leaf_step(BlrView<T> A, FactorWs<T> ws, int i, int p) {
  k_leaf_step_impl<T>(A, ws, i, p);
}

// CTA q < np: the packed LU of tile q back into the block.  CTA np + cb
// (np <= blockIdx.x < 2 np): column block cb of Linv; 2 np + cb: of Uinv (and
// of its transpose, where the caller keeps one).
template <typename T, int W>
FRANK_D void leaf_final_body(const BlrView<T>& A, const FactorWs<T>& ws, int i) {
  extern __shared__ double X[];        // b x W (ld lds)
  const int b = A.bs(i), ld = A.bmax, np = (b + W - 1) / W;
  const LeafScratch L = leaf_view<W>(ws.getrf_scratch, A.bmax);
  const int lds = leaf_lds(b);
  const int which = blockIdx.x / np, cb = blockIdx.x % np;
  if (which > 2) return;
  const int c0 = cb * W, cn = min(W, b - c0);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int jl = (np - 1) * W;                         // first row of the last panel
  const int* src = L.src + ((np - 1) & 1) * b;         // its exchanges, not yet applied to the earlier tiles
  if (which == 0) {
    T* Dp = A.dense(i, i) + (int64_t)c0 * ld;
    for (int c = wid; c < cn; c += nw)
#pragma unroll 4
      for (int r = lane; r < b; r += 32)
        Dp[r + (int64_t)c * ld] = T(L.Wm[(r >= jl && cb < np - 1 ? src[r] : r) + (int64_t)(c0 + c) * b]);
    if (threadIdx.x == 0 && cb == 0)
      atomicAdd(ws.flops + FLOP_GETRF, 2 * (unsigned long long)(2.0 / 3.0 * (double)b * b * b));
    return;
  }
  const bool lower = which == 1;
  const int rlo = lower ? c0 : 0, rhi = lower ? b : c0 + cn;   // rows that are not zero
  for (int c = wid; c < W; c += nw)
    for (int r = rlo + lane; r < rhi; r += 32) X[r + c * lds] = r == c0 + c ? 1.0 : 0.0;
  __syncthreads();
  const int g = lane >> 2, t = lane & 3;
  for (int rb = cb; lower ? rb < np : rb >= 0; rb += lower ? 1 : -1) {
    const int r0 = rb * W, rn = min(W, b - r0);
    const double* D = L.dinv + (int64_t)rb * 2 * W * W + (lower ? 0 : W * W);
    // X(rb) <- T(rb, rb)^{-1} X(rb): one 8 x 8 tile per warp and pass, all read before any is written
    constexpr int TW = W / 8;
    double acc[(TW * TW + 3) / 4][2];                   // at least four warps
    int nt = 0;
    for (int tile = wid; tile < TW * TW; tile += nw, ++nt) {
      double c1[1][1][2];
      warp_dgemm_acc<1, 1, false>(rn, cn, 0, rn, D, 1, W, X + r0, lds, 1, (tile % TW) * 8, (tile / TW) * 8, c1);
#pragma unroll
      for (int z = 0; z < (TW * TW + 3) / 4; ++z)
        if (z == nt) { acc[z][0] = c1[0][0][0]; acc[z][1] = c1[0][0][1]; }
    }
    __syncthreads();
    nt = 0;
    for (int tile = wid; tile < TW * TW; tile += nw, ++nt) {
      const int r = (tile % TW) * 8 + g, c = (tile / TW) * 8 + 2 * t;
#pragma unroll
      for (int z = 0; z < (TW * TW + 3) / 4; ++z)
        if (z == nt && r < rn) {
          if (c < cn) X[r0 + r + c * lds] = acc[z][0];
          if (c + 1 < cn) X[r0 + r + (c + 1) * lds] = acc[z][1];
        }
    }
    __syncthreads();
    // every row still to come: X(r) -= T(r, rb) X(rb)
    const int u0 = lower ? r0 + W : 0, um = lower ? b - u0 : r0;
    const int tm = (um + 31) / 32, tn = (cn + 15) / 16;
    for (int tile = wid; um > 0 && tile < tm * tn; tile += nw) {
      const int i0 = (tile % tm) * 32, j0 = (tile / tm) * 16;
      double ac[4][2][2];
      warp_dgemm_acc<4, 2, false>(um, cn, 0, rn, L.Wm + (int64_t)r0 * b, 1, b, X + r0, lds, 1, i0, j0, ac, [&](int r) {
        const int a = u0 + r;
        return lower && a >= jl && rb < np - 1 ? src[a] : a;
      });
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int r = i0 + 8 * x + g, c = j0 + 8 * y + 2 * t;
          if (r < um && c < cn) X[u0 + r + c * lds] -= ac[x][y][0];
          if (r < um && c + 1 < cn) X[u0 + r + (c + 1) * lds] -= ac[x][y][1];
        }
    }
    __syncthreads();
  }
  T* out = (lower ? ws.Linv : ws.Uinv) + (int64_t)i * ld * ld + (int64_t)c0 * ld;
  for (int c = wid; c < cn; c += nw)
    for (int r = lane; r < b; r += 32) out[r + (int64_t)c * ld] = (r >= rlo && r < rhi) ? T(X[r + c * lds]) : T(0);
  if (!lower && ws.UinvT) {
    T* outt = ws.UinvT + (int64_t)i * ld * ld + c0;
    for (int e = threadIdx.x; e < b * cn; e += blockDim.x) {
      const int c = e % cn, r = e / cn;
      outt[c + (int64_t)r * ld] = r < rhi ? T(X[r + c * lds]) : T(0);
    }
  }
}

template <typename T>
FRANK_D void k_leaf_final_impl(const BlrView<T>& A, const FactorWs<T>& ws, int i) {
  if (A.bmax <= LEAF_THREADS) leaf_final_body<T, LEAF_W>(A, ws, i);
  else leaf_final_body<T, LEAF_W_WIDE>(A, ws, i);
}

template <typename T>
__global__ void __launch_bounds__(LEAF_THREADS) k_leaf_final(BlrView<T> A, FactorWs<T> ws, int i) {
  k_leaf_final_impl<T>(A, ws, i);
}

// ---------------------------------------------------------------------------
// K2: panel of step i (trsm.cpp:92-115 with the leaf inverse; the pivots of
// K1 applied).  Task t < m: column-panel block (i+1+t, i):
//   low rank: V <- V Uinv (Vt <- Uinv^T Vt), then WL = Vt S^T;
//   dense:    A <- A Uinv.
// Task t >= m: row-panel block (i, i+1+t-m):
//   low rank: U <- Linv P U, then WU = U S;   dense: A <- Linv P A.
// Three launches, each over (task, 64-row tile of the result), so that every
// block is spread over several CTAs and no tile reads rows another tile of
// the same launch writes:
//   k_panel_gather  row tasks:    tmp = P U  (P A)                 -> WU[k]
//   k_panel_mul     column tasks: tmp = Uinv^T Vt  (A Uinv)        -> WL[ic]
//                   row tasks:    U = Linv tmp  (A = Linv tmp)
//   k_panel_fin     column tasks: Vt = tmp, then WL = Vt S^T  (A = tmp)
//                   row tasks:    WU = U S
// ---------------------------------------------------------------------------
constexpr int PANEL_THREADS = 256;
constexpr int PANEL_TILE = 64;

template <typename T>
struct PanelTask {
  bool col;      // column-panel block (else row-panel block)
  bool lr;
  int blk, rows, cols, r;   // result rows x cols (cols = rank for low rank)
  T* tmp;
};

template <typename T>
FRANK_D PanelTask<T> panel_task(const BlrView<T>& A, const FactorWs<T>& ws, int i, int t) {
  const int m = A.nb - i - 1;
  const int bi = A.bs(i), ld = A.bmax;
  PanelTask<T> P;
  P.col = t < m;
  if (P.col) {
    const int ic = i + 1 + t;
    P.blk = ic * A.nb + i;
    P.tmp = ws.WL + (int64_t)ic * ld * ld;
    P.lr = A.lslot[P.blk] >= 0;
    P.r = P.lr ? A.rank[P.blk] : 0;
    P.rows = P.lr ? bi : A.bs(ic);
    P.cols = P.lr ? P.r : bi;
  } else {
    const int k = i + 1 + (t - m);
    P.blk = i * A.nb + k;
    P.tmp = ws.WU + (int64_t)k * ld * ld;
    P.lr = A.lslot[P.blk] >= 0;
    P.r = P.lr ? A.rank[P.blk] : 0;
    P.rows = bi;
    P.cols = P.lr ? P.r : A.bs(k);
  }
  return P;
}

template <typename T>
FRANK_D T* panel_data(const BlrView<T>& A, const PanelTask<T>& P) {
  const int bi_ = P.blk / A.nb, bj_ = P.blk % A.nb;
  if (!P.lr) return A.dense(bi_, bj_);
  return P.col ? A.vt(bi_, bj_) : A.u(bi_, bj_);
}

template <typename T>
FRANK_D void k_panel_gather_impl(BlrView<T> A, FactorWs<T> ws, int i) {
  const int m = A.nb - i - 1;
  const PanelTask<T> P = panel_task(A, ws, i, m + blockIdx.x);
  const int r0 = blockIdx.y * PANEL_TILE;
  if (r0 >= P.rows) return;
  const int rn = min(PANEL_TILE, P.rows - r0), ld = A.bmax;
  const int* perm = ws.perm + (int64_t)i * ld;
  const T* src = panel_data(A, P);
  for (int e = threadIdx.x; e < rn * P.cols; e += blockDim.x) {
    const int rr = r0 + e % rn, c = e / rn;
    P.tmp[rr + (int64_t)c * ld] = src[perm[rr] + (int64_t)c * ld];
  }
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_gather(BlrView<T> A, FactorWs<T> ws, int i) {
  k_panel_gather_impl<T>(A, ws, i);
}

template <typename T>
FRANK_D void k_panel_mul_impl(BlrView<T> A, FactorWs<T> ws, int i) {
  __shared__ T gsm[2 * 16 * 64];
  const int t = blockIdx.x;
  const PanelTask<T> P = panel_task(A, ws, i, t);
  const int r0 = blockIdx.y * PANEL_TILE;
  const int bi = A.bs(i), ld = A.bmax;
  if (threadIdx.x == 0 && blockIdx.y == 0) {
    const double kk = P.lr ? P.r : (P.col ? P.rows : P.cols);
    atomicAdd(ws.flops + FLOP_PANEL, (unsigned long long)((double)bi * bi * kk));
  }
  if (r0 >= P.rows) return;
  const int rn = min(PANEL_TILE, P.rows - r0);
  T* d = panel_data(A, P);
  const T* Li = ws.Linv + (int64_t)i * ld * ld;
  const T* Ui = ws.Uinv + (int64_t)i * ld * ld;
  if (P.col) {
    if (P.lr)   // tmp(rows) = Uinv^T(rows, :) Vt
      cta_gemm<T, PANEL_THREADS>(rn, P.cols, bi, T(1), Ui + (int64_t)r0 * ld, ld, true, d, ld, false, T(0), P.tmp + r0,
                                 ld, gsm);
    else        // tmp(rows) = A(rows, :) Uinv
      cta_gemm<T, PANEL_THREADS>(rn, P.cols, bi, T(1), d + r0, ld, false, Ui, ld, false, T(0), P.tmp + r0, ld, gsm);
  } else {      // U(rows) = Linv(rows, :) P U   (A likewise)
    cta_gemm<T, PANEL_THREADS>(rn, P.cols, bi, T(1), Li + r0, ld, false, P.tmp, ld, false, T(0), d + r0, ld, gsm);
  }
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_mul(BlrView<T> A, FactorWs<T> ws, int i) {
  k_panel_mul_impl<T>(A, ws, i);
}

template <typename T>
FRANK_D void k_panel_fin_impl(BlrView<T> A, FactorWs<T> ws, int i) {
  __shared__ T gsm[2 * 16 * 64];
  const int t = blockIdx.x;
  const PanelTask<T> P = panel_task(A, ws, i, t);
  const int r0 = blockIdx.y * PANEL_TILE;
  if (r0 >= P.rows) return;
  if (!P.col && !P.lr) return;
  const int rn = min(PANEL_TILE, P.rows - r0), ld = A.bmax;
  T* d = panel_data(A, P);
  const int bi_ = P.blk / A.nb, bj_ = P.blk % A.nb;
  if (P.col) {
    for (int e = threadIdx.x; e < rn * P.cols; e += blockDim.x) {
      const int rr = r0 + e % rn, c = e / rn;
      d[rr + (int64_t)c * ld] = P.tmp[rr + (int64_t)c * ld];
    }
    __syncthreads();
    if (P.lr)   // WL(rows) = Vt(rows) S^T
      cta_gemm<T, PANEL_THREADS>(rn, P.r, P.r, T(1), d + r0, ld, false, A.s(bi_, bj_), A.kcap, true, T(0),
                                 P.tmp + r0, ld, gsm);
  } else {      // WU(rows) = U(rows) S
    cta_gemm<T, PANEL_THREADS>(rn, P.r, P.r, T(1), d + r0, ld, false, A.s(bi_, bj_), A.kcap, false, T(0),
                               P.tmp + r0, ld, gsm);
  }
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_fin(BlrView<T> A, FactorWs<T> ws, int i) {
  k_panel_fin_impl<T>(A, ws, i);
}

// Task t (0 <= t < m*(m-1)) of step i's off-diagonal targets, ordered by
// band d = |ic - k| = 1, 2, ... (the near-diagonal targets carry the largest
// ranks, so they are handed out first), within a band by row.
FRANK_D void band_task(int m, int t, int& a, int& c) {
  int d = 1;
  while (t >= 2 * (m - d)) { t -= 2 * (m - d); ++d; }
  const int half = m - d;
  if (t < half) { a = t + d; c = t; } else { a = t - half; c = t - half + d; }
}

// Next task of the step for this CTA (dynamic scheduling through an atomic
// counter; all threads receive it).
FRANK_D int next_task(int* counter, int* slot) {
  __syncthreads();
  if (threadIdx.x == 0) *slot = atomicAdd(counter, 1);
  __syncthreads();
  return *slot;
}

// Operands of the update of target (ic, k) at step i:
//   update = - XL * (WL^T WU) * YR^T,
// XL = U(ic,i) (bc x p) or dense A(ic,i) (bc x bi, WL = I),
// YR = Vt(i,k) (bk x q) or A(i,k)^T (WU = I).
template <typename T>
struct UpdOps {
  const T* XL; int p; bool left_dense;
  const T* YR; int q; bool right_dense;   // right_dense: YR^T = A(i,k) (bi x bk, ld)
  const T* WL; const T* WU;
};

template <typename T>
FRANK_D UpdOps<T> update_operands(const BlrView<T>& A, const FactorWs<T>& ws, int i, int ic, int k) {
  UpdOps<T> o;
  const int ld = A.bmax;
  const int bi = A.bs(i);
  o.WL = ws.WL + (int64_t)ic * ld * ld;
  o.WU = ws.WU + (int64_t)k * ld * ld;
  if (A.is_lr(ic, i)) { o.XL = A.u(ic, i); o.p = A.rank[ic * A.nb + i]; o.left_dense = false; }
  else { o.XL = A.dense(ic, i); o.p = bi; o.left_dense = true; }
  if (A.is_lr(i, k)) { o.YR = A.vt(i, k); o.q = A.rank[i * A.nb + k]; o.right_dense = false; }
  else { o.YR = A.dense(i, k); o.q = bi; o.right_dense = true; }
  return o;
}

// core T (p x q) = -WL^T WU, FP64, into Tm (ld p).
template <typename T>
FRANK_D void form_core(const Grp& g, const UpdOps<T>& o, int bi, int ld, double* Tm, const GrpScratch& x) {
  if (!o.left_dense && !o.right_dense) {
    g_mm(g, o.p, o.q, bi, -1.0, o.WL, ld, 1, o.WU, ld, 1, 0.0, Tm, o.p, x.part);
  } else if (!o.left_dense && o.right_dense) {
    // -WL^T (p x bi)
    for (int64_t e = threadIdx.x; e < (int64_t)o.p * o.q; e += blockDim.x) {
      const int r = e % o.p, c = e / o.p;
      Tm[e] = -double(o.WL[c + (int64_t)r * ld]);
    }
    __syncthreads();
  } else if (o.left_dense && !o.right_dense) {
    for (int64_t e = threadIdx.x; e < (int64_t)o.p * o.q; e += blockDim.x) {
      const int r = e % o.p, c = e / o.p;
      Tm[e] = -double(o.WU[r + (int64_t)c * ld]);
    }
    __syncthreads();
  } else {
    for (int64_t e = threadIdx.x; e < (int64_t)o.p * o.q; e += blockDim.x) {
      const int r = e % o.p, c = e / o.p;
      Tm[e] = (r == c) ? -1.0 : 0.0;
    }
    __syncthreads();
  }
}

template <typename T, int NT>
FRANK_D void form_core_cta(const UpdOps<T>& o, int bi, int ld, double* Tm, double* gsm) {
  if (!o.left_dense && !o.right_dense) {
    cta_gemm<double, NT>(o.p, o.q, bi, -1.0, o.WL, ld, true, o.WU, ld, false, 0.0, Tm, o.p, gsm);
    return;
  }
  for (int64_t e = threadIdx.x; e < (int64_t)o.p * o.q; e += blockDim.x) {
    const int r = e % o.p, c = e / o.p;
    if (!o.left_dense) Tm[e] = -double(o.WL[c + (int64_t)r * ld]);
    else Tm[e] = -double(o.WU[r + (int64_t)c * ld]);
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// K5: update of dense targets (diagonal blocks and inadmissible blocks):
// C += XL * T * YR^T  (gemm.cpp:180-200 for LR.LR.D; 126-178 for the others).
// One task per (target, band of band_rows rows): the band's CTA forms the
// small core T (p x q) once, X = XL(band, :) T (rows x q) in its scratch slot,
// and updates its rows of C over the full width, so the core is formed
// ceil(b / band_rows) times per target and C is streamed in full rows.
// Modes: every dense target of the step, only the next diagonal block
// (i+1, i+1) (which the next leaf getrf waits for), or all but that block.
// The next diagonal block is on the critical path and alone on the device, so
// its bands are no higher than one tile of the product (dupd_next_rows): at
// b = 256, rank 16 its launch takes 19 us, 58 in bands of 128.  Targets
// are numbered by diagonals: in row order the diagonal blocks, usually the only
// dense ones, met in the same few CTAs (m + 1 and the grid share factors).
// ---------------------------------------------------------------------------
constexpr int DUPD_THREADS = 256;
template <typename T>
FRANK_HD constexpr int dupd_next_rows() { return sizeof(T) == 8 ? 32 : 64; }
constexpr int DUPD_BAND = 128;    // rows of a dense update task (default; the autotuner may change it)
enum DenseUpdateMode { DUPD_ALL = 0, DUPD_NEXT = 1, DUPD_REST = 2 };

template <typename T>
FRANK_D void k_update_dense_impl(BlrView<T> A, FactorWs<T> ws, int i, int band_rows,
                                                                int mode) {
  __shared__ double gsm[2 * 16 * 64];
  __shared__ T gsmt[2 * 16 * 64];
  const int m = A.nb - i - 1;
  const int ld = A.bmax;
  const int bi = A.bs(i);
  double* Tm = ws.dscratch + (int64_t)blockIdx.x * ws.dscratch_stride;
  // X (rn x q, ld ldx) in the second ld x ld half of the slot: ldx * q <= ld * ld
  T* X = reinterpret_cast<T*>(Tm + (int64_t)ld * ld);
  const int bandr = min(mode == DUPD_NEXT ? min(band_rows, dupd_next_rows<T>()) : band_rows, ld);
  const int ldx = bandr;
  const int nbands = (ld + bandr - 1) / bandr;
  // pair 0 is the next diagonal block (i+1, i+1)
  const int ntask = mode == DUPD_NEXT ? nbands : m * m * nbands;
  for (int tsk = blockIdx.x; tsk < ntask; tsk += gridDim.x) {
    const int pair = tsk / nbands, band = tsk % nbands;
    if (mode == DUPD_REST && pair == 0) continue;
    const int ic = i + 1 + pair % m, k = i + 1 + (pair % m + pair / m) % m;
    if (A.is_lr(ic, k)) continue;
    const int bc = A.bs(ic), bk = A.bs(k);
    const int r0 = band * bandr;
    if (r0 >= bc) continue;
    const int rn = min(bandr, bc - r0);
    T* C = A.dense(ic, k) + r0;
    UpdOps<T> o = update_operands(A, ws, i, ic, k);
    if (threadIdx.x == 0 && band == 0)
      atomicAdd(ws.flops + FLOP_DENSE, (unsigned long long)(2.0 * bc * bk * o.q + 2.0 * bc * o.p * o.q +
                                                            2.0 * bi * o.p * o.q));
    if (o.left_dense && o.right_dense) {
      // C -= A(ic,i) A(i,k)
      cta_gemm<T, DUPD_THREADS>(rn, bk, bi, T(-1), o.XL + r0, ld, false, o.YR, ld, false, T(1), C, ld, gsmt);
      continue;
    }
    form_core_cta<T, DUPD_THREADS>(o, bi, ld, Tm, gsm);
    // X = XL(r0 : r0+rn, :) T  (rn x q), accumulate in the working precision
    cta_gemm<T, DUPD_THREADS>(rn, o.q, o.p, T(1), o.XL + r0, ld, false, Tm, o.p, false, T(0), X, ldx, gsmt);
    // C(band) += X * YR^T
    if (!o.right_dense)
      cta_gemm<T, DUPD_THREADS>(rn, bk, o.q, T(1), X, ldx, false, o.YR, ld, true, T(1), C, ld, gsmt);
    else
      cta_gemm<T, DUPD_THREADS>(rn, bk, o.q, T(1), X, ldx, false, o.YR, ld, false, T(1), C, ld, gsmt);
  }
}

template <typename T>
__global__ void __launch_bounds__(DUPD_THREADS) k_update_dense(BlrView<T> A, FactorWs<T> ws, int i, int band_rows,
                                                                int mode) {
  k_update_dense_impl<T>(A, ws, i, band_rows, mode);
}

// ---------------------------------------------------------------------------
// K4: recompression of the update into every low-rank target of the step
// (rounded LowRank addition, operations/arithmetic/addition.cpp:93-127,
// Bebendorf p.16):
//   C + W = [U_C | XL] blockdiag(S_C, T) [Vt_C | YR]^T,
//   blocked Householder QR of the stacked U bases and of the stacked V bases
//   (FP64), core M = Ru blockdiag(S_C, T) Rv^T (FP64),
//   core truncation, either
//     RRQR: truncated column-pivoted QR of M to core_scale * eps * ||M||_F,
//           then RQ of the kept rows, i.e. the reference's own fixed-accuracy
//           compressor LowRank(Dense, eps) (low_rank.cpp:50-59, geqp3.cpp:71-192)
//           applied to the core; S comes out upper triangular;
//     SVD:  one-sided Jacobi of M with the rank of find_svd_truncation_rank
//           (misc.cpp:133-146, quirk included) or the fixed rank; S diagonal;
//   new U = Qu [Q_core; 0], new V^T = Qv [V_core; 0].
// Persistent grid, one target per CTA at a time, FP64 scratch slot per CTA.
// A target is a chain of dependent column steps and short products, so the
// U side and the V side run beside each other on the two halves of the CTA
// (bases, then Q_core beside the RQ of the kept rows, then the new bases);
// the halves meet for the core and its truncation.  Panels and the core live
// in shared memory when they fit.
// ---------------------------------------------------------------------------
constexpr int RECOMP_THREADS = 512;
constexpr int SPLIT_P = 32;       // split band-1 targets whose operand rank exceeds this (default)
constexpr int SPLIT_MAX = 128;    // band-1 tasks eligible for the split (scratch slots)
constexpr int RECOMP_BMAX = 810;  // largest block order (a panel of each side in shared memory)
// Dynamic shared memory.  What it leaves of an SM's 256 KB is the L1 that the
// products' operands and the spills live on: with 226 KB the factorization of n = 8192
// at 1e-8 takes 322 ms, with 194 KB 282.  Cores up to about 141 x 141 fit with the panel
// of their RQ and take column-by-column pivoting (up to about 160 did in 226 KB, before
// that panel had to fit too); larger ones take randomized block pivoting, whose ranks
// can differ by a few at the same stopping rule.
constexpr int RECOMP_SMEM_BYTES = 194 * 1024;

struct RecompShared {
  GrpShared gs[2];               // one per half of the CTA
  unsigned long long mx[GQ + 2];
  double red[32];
  int redi[32];
  int iscr[3 * GQ];
  int flags[4];
};
constexpr int RECOMP_REGION = (RECOMP_SMEM_BYTES - (int)sizeof(RecompShared)) / 8;  // doubles for panels / core

// Panel width of the bases' QR; the panels of both sides fit side by side.
FRANK_HD int recomp_panel(int bmax) { return panel_width(bmax); }
static_assert(2 * ((RECOMP_BMAX + 15) / 16 * 16 + 4) * 8 <= RECOMP_REGION && 2 * (512 + 4) * GQ <= RECOMP_REGION,
              "panels of both sides in shared memory");

// Core of the recompression: RRQR (truncated pivoted QR + RQ of the core),
// SVD (one-sided Jacobi, find_svd_truncation_rank or the fixed rank), FAST
// (fast_rounded_addition, addition.cpp:133-189: fixed-rank targets with
// orthonormal bases; the update's bases are projected out of the target's and
// only the remainders are QR-factored; SVD core as above).
enum CoreMethod { CORE_RRQR = 0, CORE_SVD = 1, CORE_FAST = 2 };

// Scratch doubles of an svd_core whose Jacobi matrix is not in shared memory.
FRANK_HD int64_t svd_core_scratch(int mu, int mv) {
  const int64_t k = mu < mv ? mu : mv;
  return (mv + k) * k + 32 * (int64_t)mv;
}

// SVD of the recompression core Mm (mu x mv, ld ldm), preconditioned
// one-sided Jacobi: column-pivoted QR M P = Q R, then one-sided Jacobi on the
// columns of A = P R^T (mv x k) with the rotations accumulated in Z (k x k,
// appended rows); the pivoting leaves A's columns nearly orthogonal, so a few
// sweeps converge (Drmac & Veselic, "New fast and accurate Jacobi SVD
// algorithm", SIAM J. Matrix Anal. Appl. 29, 2008).
// With A Z = W S: M = (Q Z) S W^T, so the left singular vectors are Q Z (the
// QR's reflectors applied to Z) and the right ones W (the normalised columns
// of A Z); both sets are orthonormal to working accuracy whatever the
// singular value, which the next projected addition into this target relies
// on.  Tolerance plans stop the QR once the
// remaining columns are below thr = 0.01 eps ||M||_F / sqrt(mv min(mu, mv)),
// so the dropped block R22 moves the truncation test below by at most 1 % of
// its threshold.  Rank: the fixed rank of the plan, else
// find_svd_truncation_rank (misc.cpp:133-146, quirk included: the tail error
// is (min_dim - r) sigma_r^2) at ws.eps with ||M||_F as the reference norm;
// capped at kcap (counted as a rank overflow).  A core in shared memory (in_smem;
// it starts region) takes g_rrqr, a core in L2 the blocked pivoted QR.  The Jacobi matrix
// ((mv + k) x k) lies behind the core in region (cap doubles) when it
// fits, else in Atmp (global, svd_core_scratch doubles).
// tau / cnorm / partial / jpvt (mv each), sig / ord (min(mu, mv)): global.  On return
// partial[c] is the c-th largest singular value (c < r), Xo (mu x r) = U_m(:, :r)
// and Yo (mv x r) = V_m(:, :r).  Returns r (all threads).
template <typename T, int NT>
FRANK_D int svd_core(int mu, int mv, double* Mm, int ldm, bool in_smem, const FactorWs<T>& ws, int kcap,
                     double* region, int64_t cap, double* Atmp, double* tau, double* cnorm, double* partial, int* jpvt,
                     double* sig, int* ord, double* Xo, double* Yo, RecompShared& sh, int* s_rank) {
  const Grp g = grp_all();
  const int nsv = min(mu, mv);
  double f = 0.0;
  for (int e = threadIdx.x; e < mu * mv; e += blockDim.x) {
    const double v = Mm[e % mu + (int64_t)(e / mu) * ldm];
    f += v * v;
  }
  const double fro = sqrt(block_sum(f, sh.red));
  const double thr = ws.fixed_rank > 0 ? 0.0 : 0.01 * ws.eps * fro / sqrt((double)mv * (double)nsv);
  int k;
  int64_t off = 0;
  double* Qm = Mm;              // reflectors for the left vectors
  const double* stau = tau;
  int* sord = nullptr;
  if (in_smem) {
    double* st = region + (int64_t)ldm * mv;            // tau, beta / scal
    double* cand = st + 3 * nsv;
    sord = reinterpret_cast<int*>(cand + 4 * (NT / 32));
    int* at = sord + nsv;
    off = (int64_t)ldm * mv + 3 * nsv + 4 * (NT / 32) + (nsv + mv + 2) / 2;
    k = g_rrqr(g, mu, mv, Mm, ldm, thr, nsv, st, sord, at, st + nsv, cand);
    stau = st;
    const int ldj = mv + k;
    double* Aj = off + (int64_t)ldj * k <= cap ? region + off : Atmp;
    for (int e = threadIdx.x; e < ldj * k; e += blockDim.x) {
      const int c = e % ldj, j = e / ldj;
      Aj[e] = c < mv ? rrqr_r(Mm, ldm, at, j, c) : (c - mv == j ? 1.0 : 0.0);
    }
  } else {
    // a core in L2: the panel-blocked pivoted QR (F, mv x 32, in Atmp); its columns
    // are moved, so A's rows go back through jpvt
    k = cta_truncated_geqp3_blocked<NT>(mu, mv, Mm, ldm, thr, nsv, tau, cnorm, partial, jpvt, sh.red, sh.redi, Atmp,
                                        region);
    const int ldj = mv + k;
    double* Aj = (int64_t)ldj * k <= cap ? region : Atmp;
    for (int64_t e = threadIdx.x; e < (int64_t)ldj * k; e += blockDim.x) {
      const int c = e % ldj, j = e / ldj;
      if (c < mv) Aj[jpvt[c] + (int64_t)j * ldj] = c >= j ? Mm[j + (int64_t)c * ldm] : 0.0;
      else Aj[e] = c - mv == j ? 1.0 : 0.0;
    }
  }
  __syncthreads();
  const int ldj = mv + k;
  double* Aj = off + (int64_t)ldj * k <= cap ? region + off : Atmp;
  // in shared memory eight lanes a pair (more pairs at once, fewer shuffles); in
  // L2 a warp a pair, whose loads are whole lines
  const int sweeps = off + (int64_t)ldj * k <= cap ? g_jacobi(g, mv, k, Aj, ldj, 60, sh.flags, ldj)
                                                   : cta_jacobi_columns(mv, k, Aj, ldj, 60, sh.flags, ldj);
  if (sweeps < 0 && threadIdx.x == 0) atomicAdd(ws.err + ERR_JACOBI, 1);
  for (int c = threadIdx.x >> 5; c < k; c += blockDim.x >> 5) {
    double sacc = 0.0;
    for (int rr = threadIdx.x & 31; rr < mv; rr += 32) sacc += Aj[rr + (int64_t)c * ldj] * Aj[rr + (int64_t)c * ldj];
    sacc = warp_sum(sacc);
    if ((threadIdx.x & 31) == 0) sig[c] = sqrt(sacc);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    const double v = sig[c];
    int pos = 0;
    for (int d = 0; d < k; ++d) pos += sorts_before(sig[d], d, v, c);
    ord[pos] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int rr;
    if (ws.fixed_rank > 0) {
      rr = min(ws.fixed_rank, nsv);
    } else {
      // singular values beyond the k computed ones are below ||R22||, which
      // satisfies the test by the choice of thr: count them as zero
      const double thr_t = ws.eps * fro;
      rr = 0;
      double err;
      do {
        ++rr;
        err = 0.0;
        if (rr < nsv) {
          const double v = rr < k ? sig[ord[rr]] : 0.0;
          err = (double)(nsv - rr) * v * v;
        }
      } while (rr < nsv && sqrt(err) > thr_t);
    }
    if (rr > kcap) { atomicAdd(ws.err + ERR_RANK_OVERFLOW, 1); rr = kcap; }
    atomicMax(ws.err + ERR_MAX_RANK, rr);
    atomicAdd(ws.err + ERR_RECOMP, 1);
    *s_rank = rr;
  }
  __syncthreads();
  const int r = *s_rank;
  // Yo (mv x r): the columns of A Z normalised; columns beyond the computed k are zero
  for (int e = threadIdx.x; e < mv * r; e += blockDim.x) {
    const int i = e % mv, c = e / mv;
    const int src = c < k ? ord[c] : -1;
    const double sv_ = src >= 0 ? sig[src] : 0.0;
    Yo[e] = sv_ > 0.0 ? Aj[i + (int64_t)src * ldj] / sv_ : 0.0;
  }
  // Xo (mu x r) = Q [Z(:, ord); 0]
  if (in_smem) {
    const int rk = min(r, k);
    g_apply_rrqr(g, mu, k, rk, Qm, ldm, stau, sord, false, Aj + mv, ldj, ord, Xo, mu);
    for (int e = threadIdx.x; e < mu * (r - rk); e += blockDim.x) Xo[mu * rk + e] = 0.0;
  } else {
    for (int e = threadIdx.x; e < mu * r; e += blockDim.x) {
      const int i = e % mu, c = e / mu;
      Xo[e] = (i < k && c < k) ? Aj[mv + i + (int64_t)ord[c] * ldj] : 0.0;
    }
    __syncthreads();
    cta_apply_q(mu, k, Mm, ldm, tau, r, Xo, (int64_t)mu);
  }
  // the kept singular values in order, in partial (free after the QR)
  for (int c = threadIdx.x; c < r; c += blockDim.x) partial[c] = c < k ? sig[ord[c]] : 0.0;
  __syncthreads();
  return r;
}

// Leading dimension of a side's scratch: 16-byte aligned columns, as in shared
// memory, so that the products take the same loads and sums in both (a split
// target has twice the shared memory for a side).
FRANK_HD int side_ld(int rows) { return (rows + 1) & ~1; }

struct RecompLayout {
  int64_t ash, bsh, t, gu, gv, mtmp, mglob, y1, tv, tfu, tfv, tfc, tfr, om, w, part, tau_c, sig, cn, pn, jp, ji, total;
};

FRANK_HD RecompLayout recomp_layout(int bmax, int smax) {
  RecompLayout L;
  int64_t o = 0;
  auto take = [&](int64_t n) { int64_t r = o; o += (n + 31) & ~int64_t(31); return r; };
  const int mu = smax < bmax ? smax : bmax;
  const int64_t np = bmax / recomp_panel(bmax) + 1;
  L.ash = take((int64_t)side_ld(bmax) * smax);
  L.bsh = take((int64_t)side_ld(bmax) * smax);
  L.t = take((int64_t)bmax * bmax);
  L.gu = take((int64_t)mu * smax);
  L.gv = take((int64_t)mu * smax);
  L.mtmp = take((int64_t)mu * smax);
  const int64_t svd = svd_core_scratch(mu, mu), sq = (int64_t)mu * mu;
  L.mglob = take(sq);
  L.y1 = take(sq);
  L.tv = take(svd > (int64_t)bmax * mu ? svd : (int64_t)bmax * mu);
  L.tfu = take(np * GQ * GQ);
  L.tfv = take(np * GQ * GQ);
  L.tfc = take((mu / 8 + 2) * (int64_t)GQ * GQ);
  L.tfr = take((mu / 8 + 2) * (int64_t)GQ * GQ);
  L.om = take((GQ + 8) * (int64_t)mu);
  L.w = take(4 * (int64_t)GQ * (smax > bmax ? smax : bmax));
  L.part = take(2 * (int64_t)G_PART);
  L.tau_c = take(mu);
  L.sig = take(mu);
  L.cn = take(mu);
  L.pn = take(mu);
  L.jp = take(mu);
  L.ji = take(mu);
  L.total = o;
  return L;
}

// One target's operands and scratch, in shared memory: the phases below are
// long and inlined, and values kept in registers across all of them would
// spill to local memory, which beside RECOMP_SMEM_BYTES has some 30 KB of L1.
template <typename T>
struct RecompSide {
  const T* X;                  // update basis (XL or YR)
  T* C;                        // the target's basis
  double *S, *G, *Tf, *Tn, *Z2;
  GrpScratch x;
  int bb, pp, mm, xt;          // rows, update rank, core dimension, X transposed
};

template <typename T>
struct RecompTask {
  RecompSide<T> s[2];
  UpdOps<T> o;
  double *base, *Tm, *Mtmp, *Mg, *Y1;
  T* Sc;
  int blk, kc, mu, mv, proj, side, tsk, ok;
};

template <typename T>
FRANK_D void k_recompress_impl(const BlrView<T>& A, const FactorWs<T>& ws, int i, int smax,
                                                               int core_method, double core_scale,
                                                               int only_dense_operands, int* counter, int nsplit,
                                                               double* split_base, int* split_done, int proj_tol,
                                                               int split_p, int core_smem) {
  extern __shared__ double dsm[];
  RecompShared& sh = *reinterpret_cast<RecompShared*>(dsm);
  double* region = dsm + sizeof(RecompShared) / 8;
  __shared__ int s_rank, s_last, s_task;
  __shared__ RecompTask<T> tk;
  const int hf = threadIdx.x >= RECOMP_THREADS / 2;
  const int lane = threadIdx.x & 31;
  for (;;) {
    const int q = next_task(counter, &s_task);
    // Split targets: band-1 targets (the first 2(m-1) tasks, largest ranks)
    // whose operands have ranks above SPLIT_P get one task per side of the
    // bases' QR, run on two CTAs into the target's own scratch slot;
    // the CTA that finishes second does the rest (no waiting).  The test uses
    // only operand ranks, which no CTA changes during the launch.
    {
      const int m = A.nb - i - 1;
      const int nspl = split_base ? min(nsplit, 2 * (m - 1)) : 0;
      if (q >= 2 * nspl + m * (m - 1)) break;
      if (threadIdx.x == 0) {
        const int side = q < 2 * nspl ? (q & 1) : -1;
        const int tsk = q < 2 * nspl ? (q >> 1) : q - 2 * nspl;
        int a_, c_;
        band_task(m, tsk, a_, c_);
        const int ic = i + 1 + a_, k = i + 1 + c_;
        const bool ll = A.is_lr(ic, i), lr = A.is_lr(i, k);
        const bool split_t = tsk < nspl && split_p > 0 && ll && lr &&
                             max(A.rank[ic * A.nb + i], A.rank[i * A.nb + k]) > split_p;
        tk.ok = A.is_lr(ic, k) && !(only_dense_operands && ll && lr) && (side >= 0) == split_t;
        if (tk.ok) {
          tk.o = update_operands(A, ws, i, ic, k);
          tk.blk = ic * A.nb + k;
          tk.kc = A.rank[tk.blk];
          tk.side = side;
          tk.tsk = tsk;
          const int bc = A.bs(ic), bk = A.bs(k), kc = tk.kc, su = kc + tk.o.p, sv = kc + tk.o.q;
          if (su > smax || sv > smax) {
            atomicAdd(ws.err + ERR_BOUNDS, 1);
            tk.ok = 0;
          }
          // Bases.  Stacked (rounded_addition, addition.cpp:93-127): Householder QR
          // of [U_C | U_B] and of [V_C | V_B].  Projected (fast_rounded_addition,
          // addition.cpp:133-189, the default of fixed-rank plans, and on request
          // for tolerance plans): U_C and V_C have orthonormal columns (every
          // target comes from construction, a core SVD / RRQR or the reset
          // truncation), so U_B is projected out of span(U_C) twice, Zu = U_C^T U_B,
          // and only the remainder Y_u = U_B - U_C Zu is QR-factored; the same on the
          // V side.  Both give the same sum C + B = [U_C | Q] M [V_C | Q']^T.
          tk.proj = (core_method == CORE_FAST ? ws.fixed_rank > 0 : proj_tol != 0) && kc > 0 && tk.o.p > 0 &&
                    tk.o.q > 0 && !tk.o.left_dense && !tk.o.right_dense && su <= bc && sv <= bk;
          tk.mu = tk.proj ? su : min(bc, su);
          tk.mv = tk.proj ? sv : min(bk, sv);
          const RecompLayout L = recomp_layout(A.bmax, smax);
          double* base = side >= 0 ? split_base + (int64_t)tsk * ws.rscratch_stride
                                   : ws.rscratch + (int64_t)blockIdx.x * ws.rscratch_stride;
          tk.base = base;
          tk.Tm = base + L.t; tk.Mtmp = base + L.mtmp; tk.Mg = base + L.mglob; tk.Y1 = base + L.y1;
          tk.Sc = A.s(ic, k);
          const int64_t wstep = (int64_t)GQ * max(smax, A.bmax);
          for (int sd = 0; sd < 2; ++sd) {
            RecompSide<T>& d = tk.s[sd];
            d.X = sd ? tk.o.YR : tk.o.XL;
            d.C = sd ? A.vt(ic, k) : A.u(ic, k);
            d.S = base + (sd ? L.bsh : L.ash);
            d.G = base + (sd ? L.gv : L.gu);
            d.Tf = base + (sd ? L.tfv : L.tfu);
            d.Tn = base + (sd ? L.tv : L.t);
            d.Z2 = base + (sd ? L.mglob : L.mtmp);
            d.x = GrpScratch{base + L.w + 2 * sd * wstep, base + L.w + (2 * sd + 1) * wstep,
                             base + L.part + sd * (int64_t)G_PART};
            d.bb = sd ? bk : bc;
            d.pp = sd ? tk.o.q : tk.o.p;
            d.mm = sd ? tk.mv : tk.mu;
            d.xt = sd && tk.o.right_dense;     // A(i,k)^T
          }
        }
      }
      __syncthreads();
      if (!tk.ok) continue;
    }
    const int ld = A.bmax, wp = recomp_panel(A.bmax);
    if (tk.side != 1) form_core(grp_all(), tk.o, A.bs(i), ld, tk.Tm, tk.s[0].x);
    {
      // one side's basis per half (both halves on one side of a split target):
      // projected, [Zu; Ru] (su x p) in G and the clean V of the remainder's
      // QR in S; stacked, R (mu x su) in G and V in S
      const int sd = tk.side >= 0 ? tk.side : hf;
      const Grp g = tk.side >= 0 ? grp_all() : grp_half(hf);
      const RecompSide<T>& d = tk.s[sd];
      double* smP = region + (tk.side >= 0 ? 0 : hf * (RECOMP_REGION / 2));
      const int kc = tk.kc, bb = d.bb, cols = tk.proj ? d.pp : kc + d.pp;
      // the whole side in shared memory where it fits, else panel by panel
      const bool sm = panel_ld(bb) * cols <= (tk.side >= 0 ? RECOMP_REGION : RECOMP_REGION / 2);
      double* Y = sm ? smP : d.S;
      const int ldy = sm ? panel_ld(bb) : side_ld(bb);
      for (int c = g.wid; c < cols; c += g.nw) {
        const int cx = tk.proj ? c : c - kc;
        const T* src = cx < 0 ? d.C + (int64_t)c * ld : d.X + (d.xt ? (int64_t)cx : (int64_t)cx * ld);
        const int step = cx >= 0 && d.xt ? ld : 1;
#pragma unroll 4
        for (int r = lane; r < bb; r += 32) Y[r + (int64_t)c * ldy] = double(src[(int64_t)r * step]);
      }
      g.sync();
      if (tk.proj) g_project_out(g, bb, kc, d.pp, (const T*)d.C, 1, ld, Y, ldy, d.G, kc + d.pp, d.Z2, d.x);
      g_qr(g, bb, cols, Y, ldy, d.S, side_ld(bb), d.G + (tk.proj ? kc : 0), tk.proj ? kc + d.pp : d.mm, d.Tf, wp,
           sm ? nullptr : smP, sh.gs[sd], d.x);
    }
    __syncthreads();
    if (tk.side >= 0) {
      // publish this side; the second of the two CTAs goes on with the target
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) s_last = atomicAdd(split_done + tk.tsk, 1);
      __syncthreads();
      if (s_last == 0) continue;
      __threadfence();
    }
    // Core M (mu x mv), in shared memory if it fits with the panel of its RQ and is not above the tuned size
    // (small cores always: the L2 path works on panels of its own).
    // Projected: M = [I Zu; 0 Ru] blockdiag(S_C, T) [I Zv; 0 Rv']^T = [Zu; Ru] T [Zv; Rv']^T + S_C;
    // stacked: M = [Ru(:, :kc) S_C | Ru(:, kc:) T] Rv^T.
    const int mu = tk.mu, mv = tk.mv, mn = min(mu, mv);
    const int core_need = rrqr_ld(mu) * mv + 3 * mn + 4 * (RECOMP_THREADS / 32) + (mn + mv + 2) / 2;
    const bool in_smem = core_need + 8 * panel_ld(mv) <= RECOMP_REGION && mu <= G_COLS_MAX &&
                         (mu < 64 || core_need <= core_smem);
    double* const Mm = in_smem ? region : tk.Mg;
    const int ldm = in_smem ? rrqr_ld(mu) : mu;
    {
      const Grp all = grp_all();
      const int kc = tk.kc, p = tk.o.p, qq = tk.o.q;
      const double *Gu = tk.s[0].G, *Gv = tk.s[1].G;
      if (!tk.proj) {
        // S_C in FP64 (Y1 is free)
        for (int e = threadIdx.x; e < kc * kc; e += blockDim.x)
          tk.Y1[e] = double(tk.Sc[e % kc + (int64_t)(e / kc) * A.kcap]);
        __syncthreads();
      }
      // projected: Mtmp = Gu T, M = Mtmp Gv^T; stacked: the two parts of Mtmp first
      for (int op = tk.proj ? 1 : 0; op < 3; ++op) {
        const double* a = op == 2 ? tk.Mtmp : Gu + (op == 1 && !tk.proj ? (int64_t)kc * mu : 0);
        const double* b = op == 0 ? tk.Y1 : (op == 1 ? tk.Tm : Gv);
        double* c = op == 2 ? Mm : tk.Mtmp + (op == 1 && !tk.proj ? (int64_t)kc * mu : 0);
        const int kk = op == 0 ? kc : (op == 1 ? p : (tk.proj ? qq : kc + qq));
        g_mm(all, mu, op == 0 ? kc : (op == 1 ? qq : mv), kk, 1.0, a, 1, mu, b, op == 2 ? 1 : kk, op == 2 ? mv : 1,
             0.0, c, op == 2 ? ldm : mu, tk.s[0].x.part);
      }
      if (tk.proj) {
        for (int e = threadIdx.x; e < kc * kc; e += blockDim.x)
          Mm[e % kc + (e / kc) * ldm] += double(tk.Sc[e % kc + (int64_t)(e / kc) * A.kcap]);
        __syncthreads();
      }
    }
    int r = 0;
    double* const X1 = tk.s[0].G;     // Q_core (mu x r); G is free once the core is formed
    if (core_method == CORE_RRQR && ws.fixed_rank == 0) {
      // shared-memory vectors of the pivoted QR, behind the core
      double* tau = region + rrqr_ld(mu) * mv;
      double* cand = tau + 3 * mn;
      int* ord = reinterpret_cast<int*>(cand + 4 * (RECOMP_THREADS / 32));
      int* at = ord + mn;
      const RecompLayout L = recomp_layout(A.bmax, smax);
      int* jpvt = reinterpret_cast<int*>(tk.base + L.jp);
      // panel width of the L2 path: its sketch and its panel fit shared memory
      int wc = panel_width(mu);
      while (wc > 8 && rand_qrcp_smem(mu, mv, wc) > RECOMP_REGION) wc -= 8;
      {
        double f = 0.0;
        for (int e = threadIdx.x; e < mu * mv; e += blockDim.x) {
          const double v = Mm[e % mu + (e / mu) * ldm];
          f += v * v;
        }
        const double thr = core_scale * ws.eps * sqrt(block_sum(f, sh.red));
        if (in_smem)
          r = g_rrqr(grp_all(), mu, mv, Mm, ldm, thr, A.kcap, tau, ord, at, tau + mn, cand);
        else
          r = g_rand_qrcp(grp_all(), mu, mv, Mm, ldm, tk.s[1].G, mu, thr, A.kcap, wc, jpvt, tk.base + L.tfc,
                          tk.base + L.om, tk.base + L.cn, region, sh.iscr, sh.mx, sh.gs[0], tk.s[0].x);
      }
      if (threadIdx.x == 0) {
        if (r >= A.kcap && r < mn) atomicAdd(ws.err + ERR_RANK_OVERFLOW, 1);
        atomicMax(ws.err + ERR_MAX_RANK, max(r, 1));
        atomicAdd(ws.err + ERR_RECOMP, 1);
      }
      if (r == 0) {
        // zero core: rank-1 zero block (geqp3.cpp:97-102)
        for (int sd = 0; sd < 2; ++sd)
          for (int e = threadIdx.x; e < tk.s[sd].bb; e += blockDim.x) tk.s[sd].C[e] = T(e == 0 ? 1.0 : 0.0);
        if (threadIdx.x == 0) { tk.Sc[0] = T(0); A.rank[tk.blk] = 1; }
        __syncthreads();
        continue;
      }
      // half 0: X1 = Q_core(:, :r).  Half 1: RQ of the kept rows R P^T = S Q', by the
      // QR of X2 (mv x r) = (R P^T)^T J: S = J Rt^T J, and its explicit Q in Qt.
      const Grp half = grp_half(hf);
      double* const X2 = tk.Mtmp;
      double* const Qt = tk.s[1].G;            // after the rows of R of an L2 core have been read
      const int w2 = min(panel_width(mv), (RECOMP_REGION - (in_smem ? core_need : 0)) / panel_ld(mv));
      if (hf == 1) {
        for (int e = half.tid; e < mv * r; e += half.nt) {
          const int c = e % mv, row = r - 1 - e / mv;
          if (in_smem) X2[e] = rrqr_r(Mm, ldm, at, row, c);
          else X2[jpvt[c] + (e / mv) * mv] = row <= c ? tk.s[1].G[row + (int64_t)c * mu] : 0.0;
        }
        half.sync();
        double* Rt = tk.Y1;                    // r x r
        g_qr(half, mv, r, X2, mv, X2, mv, Rt, r, tk.base + L.tfr, w2, in_smem ? region + core_need : region,
             sh.gs[1], tk.s[1].x);
        for (int e = half.tid; e < r * r; e += half.nt) {
          const int a = e % r, c = e / r;
          const int ra = r - 1 - c, ca = r - 1 - a;
          tk.Sc[a + (int64_t)c * A.kcap] = T(ra <= ca ? Rt[ra + ca * r] : 0.0);
        }
      } else if (in_smem) {
        g_apply_rrqr(half, mu, r, r, Mm, ldm, tau, ord, true, nullptr, 0, nullptr, X1, mu);
      }
      // explicit factors by blocked application: Qt, and X1 of a core in L2
      if (hf == 1 || !in_smem) {
        double* X = hf ? Qt : X1;
        const int mm = hf ? mv : mu;
        for (int e = half.tid; e < mm * r; e += half.nt) X[e] = (e % mm) == (e / mm) ? 1.0 : 0.0;
        half.sync();
        g_apply_q(half, mm, r, hf ? X2 : Mm, mm, tk.base + (hf ? L.tfr : L.tfc), hf ? w2 : wc, r, X, mm, r,
                  tk.s[hf].x);
        if (hf == 1)
          for (int e = half.tid; e < mv * r; e += half.nt) tk.Y1[e] = Qt[e % mv + (r - 1 - e / mv) * mv];
      }
      __syncthreads();
    } else {
      const RecompLayout L = recomp_layout(A.bmax, smax);
      double* pn = tk.base + L.pn;
      r = svd_core<T, RECOMP_THREADS>(mu, mv, Mm, ldm, in_smem, ws, A.kcap, region, RECOMP_REGION, tk.base + L.tv,
                                      tk.base + L.tau_c, tk.base + L.cn, pn, reinterpret_cast<int*>(tk.base + L.jp),
                                      tk.base + L.sig, reinterpret_cast<int*>(tk.base + L.ji), X1, tk.Y1, sh, &s_rank);
      for (int e = threadIdx.x; e < r * r; e += blockDim.x)
        tk.Sc[e % r + (int64_t)(e / r) * A.kcap] = T(e % r == e / r ? pn[e / r] : 0.0);
      __syncthreads();
    }
    {
      // new bases, a side per half.  Stacked: U = Qu [X1; 0]; projected:
      // U = [U_C | Q_u] X1 = Q_u [X1(kc:); 0] + U_C X1(:kc), in FP64 scratch
      // (U_C is an operand, so the block itself is written last)
      const Grp half = grp_half(hf);
      const RecompSide<T>& d = tk.s[hf];
      const double* X = hf ? tk.Y1 : X1;
      const int bb = d.bb, mm = d.mm, skip = tk.proj ? tk.kc : 0, refl = tk.proj ? d.pp : mm;
      for (int c = half.wid; c < r; c += half.nw)
#pragma unroll 4
        for (int e = lane; e < bb; e += 32) d.Tn[e + c * bb] = e < refl ? X[skip + e + c * mm] : 0.0;
      half.sync();
      g_apply_q(half, bb, refl, d.S, side_ld(bb), d.Tf, wp, r, d.Tn, bb, refl, d.x);
      if (tk.proj) g_mm(half, bb, r, skip, 1.0, (const T*)d.C, 1, ld, X, mm, 1, 1.0, d.Tn, bb, d.x.part);
      for (int c = half.wid; c < r; c += half.nw)
#pragma unroll 4
        for (int e = lane; e < bb; e += 32) d.C[e + (int64_t)c * ld] = T(d.Tn[e + c * bb]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int bc = tk.s[0].bb, bk = tk.s[1].bb, bi = A.bs(i);
      atomicAdd(ws.flops + FLOP_RECOMP,
                (unsigned long long)(tk.proj ? fast_rounded_addition_flops(bc, bk, bi, tk.kc, tk.o.p, tk.o.q, r)
                                             : rounded_addition_flops(bc, bk, bi, tk.kc, tk.o.p, tk.o.q, r)));
      A.rank[tk.blk] = r;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(RECOMP_THREADS) k_recompress(BlrView<T> A, FactorWs<T> ws, int i, int smax,
                                                               int core_method, double core_scale,
                                                               int only_dense_operands, int* counter, int nsplit,
                                                               double* split_base, int* split_done, int proj_tol,
                                                               int split_p, int core_smem) {
  k_recompress_impl<T>(A, ws, i, smax, core_method, core_scale, only_dense_operands, counter, nsplit, split_base,
                       split_done, proj_tol, split_p, core_smem);
}

// ---------------------------------------------------------------------------
// K4' (mixed path): recompression by Gram matrices.  Same update and the same
// core truncation (RRQR + RQ of the core, or its fixed rank) as k_recompress,
// but the stacked bases A = [U_C | U_L] and B = [Vt_C | V_U] are not
// factored along their b rows: their FP64 Gram matrices A^T A, B^T B (one
// GEMM pass over the FP32 bases) are factored by pivoted Cholesky,
// A Pa ~= Qa [Ra11 Ra12] with Qa = A Pa(:, :ra) Ra11^{-1}, dropping directions
// whose relative norm is below sqrt(gram_tol); the core is
// M = Ra Pa^T blockdiag(S_C, T) Pb Rb^T and the new bases are
// U = A Pa [Ra11^{-1} Q_core; 0], V^T = B Pb [Rb11^{-1} V_core; 0].
// A Gram matrix in FP64 resolves directions down to ~1e-8 of the basis norm,
// which is ample for the loose factor tolerance of the mixed path (the FP64
// path keeps the Householder kernel).  Targets with a dense operand are left
// to k_recompress.  256 threads; small matrices in shared memory when they fit.
// ---------------------------------------------------------------------------
constexpr int GRAM_THREADS = 256;
constexpr int GRAM_SMEM_BYTES = 110 * 1024;
constexpr int GRAM_REGION = GRAM_SMEM_BYTES / 8;

// Per-CTA global scratch of the Gram kernel (used for the small matrices when
// they do not fit shared memory, and for the tall outputs).
struct GramLayout {
  int64_t ga, gb, m1, m2, m3, m4, vec, uo, vo, tm, total;
};

FRANK_HD GramLayout gram_layout(int bmax, int smax) {
  GramLayout L;
  int64_t o = 0;
  auto take = [&](int64_t n) { int64_t r = o; o += (n + 31) & ~int64_t(31); return r; };
  L.ga = take((int64_t)smax * smax);
  L.gb = take((int64_t)smax * smax);
  L.m1 = take((int64_t)smax * smax);
  L.m2 = take((int64_t)smax * smax);
  L.m3 = take((int64_t)smax * smax);
  L.m4 = take((int64_t)smax * smax);
  L.vec = take(16 * (int64_t)smax);
  L.uo = take((int64_t)bmax * smax);
  L.vo = take((int64_t)bmax * smax);
  L.tm = take((int64_t)bmax * bmax);
  L.total = o;
  return L;
}

template <typename T>
__global__ void __launch_bounds__(GRAM_THREADS) k_recompress_gram(BlrView<T> A, FactorWs<T> ws, int i, int smax,
                                                                  double core_scale, double gram_tol, int* counter) {
  extern __shared__ double region[];
  __shared__ double gsm[2 * 16 * 64];
  __shared__ double red[32];
  __shared__ int s_redi[32];
  __shared__ int s_r[3];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int m = A.nb - i - 1;
  const int ld = A.bmax;
  const int bi = A.bs(i);
  const GramLayout L = gram_layout(A.bmax, smax);
  double* base = ws.rscratch + (int64_t)blockIdx.x * ws.rscratch_stride;
  __shared__ int s_task;
  const int ntask = m * (m - 1);
  for (int tsk = next_task(counter, &s_task); tsk < ntask; tsk = next_task(counter, &s_task)) {
    int a_, c_;
    band_task(m, tsk, a_, c_);
    const int ic = i + 1 + a_, k = i + 1 + c_;
    if (!A.is_lr(ic, k) || !A.is_lr(ic, i) || !A.is_lr(i, k)) continue;
    const int blk = ic * A.nb + k;
    const int bc = A.bs(ic), bk = A.bs(k);
    const int kc = A.rank[blk];
    const int p = A.rank[ic * A.nb + i], q = A.rank[i * A.nb + k];
    const int su = kc + p, sv = kc + q;
    if (su > smax || sv > smax) {
      if (threadIdx.x == 0) atomicAdd(ws.err + ERR_BOUNDS, 1);
      continue;
    }
    const T* Uc = A.u(ic, k);
    const T* Sc = A.s(ic, k);
    const T* Vc = A.vt(ic, k);
    const T* UL = A.u(ic, i);
    const T* VU = A.vt(i, k);
    const T* WL = ws.WL + (int64_t)ic * ld * ld;
    const T* WU = ws.WU + (int64_t)k * ld * ld;
    const int sm_ = su > sv ? su : sv;
    // small matrices: Ga (su^2), Gb (sv^2), M1, M2 (su*sv), M3, M4 (sv*sv), vec;
    // all in shared memory when they fit (then also the V-side temporaries)
    const int64_t sq = (int64_t)sm_ * sm_;
    const int64_t need = 6 * sq + 16 * (int64_t)sm_;
    const bool in_sm = need <= GRAM_REGION;
    double *Ga, *Gb, *M1, *M2, *M3, *M4, *vec;
    if (in_sm) {
      Ga = region; Gb = Ga + sq; M1 = Gb + sq; M2 = M1 + sq; M3 = M2 + sq; M4 = M3 + sq; vec = M4 + sq;
    } else {
      Ga = base + L.ga; Gb = base + L.gb; M1 = base + L.m1; M2 = base + L.m2; M3 = base + L.m3; M4 = base + L.m4;
      vec = base + L.vec;
    }
    int* pa = reinterpret_cast<int*>(vec);
    int* pb = pa + sm_;
    int* jp = pb + sm_;
    int* ji = jp + sm_;
    double* tc = vec + 2 * (int64_t)sm_;
    double* cn = tc + sm_;
    double* pn = cn + sm_;
    double* tc2 = pn + sm_;
    double* Tm = base + L.tm;
    double* Uo = base + L.uo;
    double* Vo = base + L.vo;
    // small targets: warp-level factorizations in shared memory; large ones:
    // CTA-level factorizations
    const bool small = in_sm && su <= 64 && sv <= 64;
    // T = -WL^T WU (p x q); Gram matrices of the stacked bases (upper blocks)
    // skinny products: warp dot products when small, tiled GEMM otherwise
    auto tn = [&](int mm_, int nn_, int kk_, double al, const T* Ap, const T* Bp, double* Cp, int ldc_) {
      if ((int64_t)mm_ * nn_ <= 1024) cta_gemm_tn_dot(mm_, nn_, kk_, al, Ap, ld, Bp, ld, Cp, ldc_);
      else cta_gemm<double, GRAM_THREADS>(mm_, nn_, kk_, al, Ap, ld, true, Bp, ld, false, 0.0, Cp, ldc_, gsm);
    };
    tn(p, q, bi, -1.0, WL, WU, Tm, p);
    tn(kc, kc, bc, 1.0, Uc, Uc, Ga, su);
    tn(kc, p, bc, 1.0, Uc, UL, Ga + (int64_t)kc * su, su);
    tn(p, p, bc, 1.0, UL, UL, Ga + kc + (int64_t)kc * su, su);
    tn(kc, kc, bk, 1.0, Vc, Vc, Gb, sv);
    tn(kc, q, bk, 1.0, Vc, VU, Gb + (int64_t)kc * sv, sv);
    tn(q, q, bk, 1.0, VU, VU, Gb + kc + (int64_t)kc * sv, sv);
    for (int e = threadIdx.x; e < kc * p; e += blockDim.x) {
      const int r = e % kc, c = e / kc;
      Ga[(kc + c) + (int64_t)r * su] = Ga[r + (int64_t)(kc + c) * su];
    }
    for (int e = threadIdx.x; e < kc * q; e += blockDim.x) {
      const int r = e % kc, c = e / kc;
      Gb[(kc + c) + (int64_t)r * sv] = Gb[r + (int64_t)(kc + c) * sv];
    }
    __syncthreads();
    // pivoted Cholesky of both Gram matrices (one warp each when small)
    if (small) {
      if (wid == 0) {
        const int r_ = warp_pivoted_cholesky(su, Ga, su, pa, gram_tol, su);
        if (lane == 0) s_r[0] = r_;
      } else if (wid == 1) {
        const int r_ = warp_pivoted_cholesky(sv, Gb, sv, pb, gram_tol, sv);
        if (lane == 0) s_r[1] = r_;
      }
    } else {
      const int r0 = cta_pivoted_cholesky(su, Ga, su, pa, gram_tol, su, red, s_redi);
      const int r1 = cta_pivoted_cholesky(sv, Gb, sv, pb, gram_tol, sv, red, s_redi);
      if (threadIdx.x == 0) { s_r[0] = r0; s_r[1] = r1; }
    }
    __syncthreads();
    const int ra = s_r[0], rb = s_r[1];
    // M1 = Pa^T blockdiag(S_C, T) Pb (su x sv); zero the lower parts of Ra, Rb
    for (int64_t e = threadIdx.x; e < (int64_t)su * sv; e += blockDim.x) {
      const int r = e % su, c = e / su;
      const int orr = pa[r], occ = pb[c];
      double v = 0.0;
      if (orr < kc && occ < kc) v = double(Sc[orr + (int64_t)occ * A.kcap]);
      else if (orr >= kc && occ >= kc) v = Tm[(orr - kc) + (int64_t)(occ - kc) * p];
      M1[e] = v;
    }
    for (int64_t e = threadIdx.x; e < (int64_t)ra * su; e += blockDim.x) {
      const int r = e % ra, c = e / ra;
      if (r > c) Ga[r + (int64_t)c * su] = 0.0;
    }
    for (int64_t e = threadIdx.x; e < (int64_t)rb * sv; e += blockDim.x) {
      const int r = e % rb, c = e / rb;
      if (r > c) Gb[r + (int64_t)c * sv] = 0.0;
    }
    __syncthreads();
    // M2 (ra x sv) = Ra M1 ; Core = M1 <- M2 Rb^T (ra x rb)
    for (int64_t e = threadIdx.x; e < (int64_t)ra * sv; e += blockDim.x) {
      const int r = e % ra, c = e / ra;
      double acc = 0.0;
      for (int t = r; t < su; ++t) acc += Ga[r + (int64_t)t * su] * M1[t + (int64_t)c * su];
      M2[e] = acc;
    }
    __syncthreads();
    double* Core = M1;  // ra x rb, ld ra
    for (int64_t e = threadIdx.x; e < (int64_t)ra * rb; e += blockDim.x) {
      const int r = e % ra, c = e / ra;
      double acc = 0.0;
      for (int t = c; t < sv; ++t) acc += M2[r + (int64_t)t * ra] * Gb[c + (int64_t)t * sv];
      Core[e] = acc;
    }
    double f = 0.0;
    __syncthreads();
    for (int64_t e = threadIdx.x; e < (int64_t)ra * rb; e += blockDim.x) f += Core[e] * Core[e];
    f = block_sum(f, red);
    const double thr = ws.fixed_rank > 0 ? 0.0 : core_scale * ws.eps * sqrt(f);
    const int maxr = ws.fixed_rank > 0 ? min(ws.fixed_rank, A.kcap) : A.kcap;
    if (small) {
      if (wid == 0) {
        const int r_ = (ra > 0 && rb > 0) ? warp_truncated_geqp3(ra, rb, Core, ra, thr, maxr, tc, cn, pn, jp) : 0;
        if (lane == 0) s_r[2] = r_;
      }
    } else {
      const int r_ = (ra > 0 && rb > 0) ? cta_truncated_geqp3(ra, rb, Core, ra, thr, maxr, tc, cn, pn, jp, red, s_redi)
                                        : 0;
      if (threadIdx.x == 0) s_r[2] = r_;
    }
    __syncthreads();
    const int r = s_r[2];
    if (r == 0) {
      T* Uw = A.u(ic, k); T* Vw = A.vt(ic, k); T* Sw = A.s(ic, k);
      for (int e = threadIdx.x; e < bc; e += blockDim.x) Uw[e] = T(e == 0 ? 1.0 : 0.0);
      for (int e = threadIdx.x; e < bk; e += blockDim.x) Vw[e] = T(e == 0 ? 1.0 : 0.0);
      if (threadIdx.x == 0) { Sw[0] = T(0); A.rank[blk] = 1; atomicAdd(ws.err + ERR_RECOMP, 1); }
      __syncthreads();
      continue;
    }
    if (threadIdx.x == 0) {
      if (ws.fixed_rank == 0 && r >= A.kcap && r < min(ra, rb)) atomicAdd(ws.err + ERR_RANK_OVERFLOW, 1);
      atomicMax(ws.err + ERR_MAX_RANK, r);
      atomicAdd(ws.err + ERR_RECOMP, 1);
      atomicAdd(ws.flops + FLOP_RECOMP, (unsigned long long)rounded_addition_flops(bc, bk, bi, kc, p, q, r));
    }
    double* X1 = M2;   // ra x r (M2 no longer needed)
    double* X2 = M3;   // rb x r
    double* Qt = M4;   // rb x r
    double* Yk = M4;   // Qt with its columns reversed in place
    T* Sw = A.s(ic, k);
    if (small) {
      if (wid == 0) {
        // X1 = Ra11^{-1} Q_core
        for (int e = lane; e < ra * r; e += 32) X1[e] = ((e % ra) == (e / ra)) ? 1.0 : 0.0;
        __syncwarp();
        warp_apply_q(ra, r, Core, ra, tc, r, X1, ra);
        warp_upper_solve(ra, Ga, su, r, X1, ra);
      } else if (wid == 1) {
        // RQ of the kept rows R_core Pcore^T (r x rb): QR of X2 = (R_perm)^T J
        for (int c = lane; c < rb; c += 32) ji[jp[c]] = c;
        __syncwarp();
        for (int e = lane; e < rb * r; e += 32) {
          const int c = e % rb, a = e / rb;
          const int row = r - 1 - a, src = ji[c];
          X2[e] = (row <= src) ? Core[row + (int64_t)src * ra] : 0.0;
        }
        __syncwarp();
        warp_householder_qr(rb, r, X2, rb, tc2);
        for (int e = lane; e < r * r; e += 32) {
          const int a = e % r, c = e / r;
          const int ra_ = r - 1 - c, ca = r - 1 - a;
          Sw[a + (int64_t)c * A.kcap] = T((ra_ <= ca) ? X2[ra_ + (int64_t)ca * rb] : 0.0);
        }
        for (int e = lane; e < rb * r; e += 32) Qt[e] = ((e % rb) == (e / rb)) ? 1.0 : 0.0;
        __syncwarp();
        warp_apply_q(rb, r, X2, rb, tc2, r, Qt, rb);
        for (int e = lane; e < rb * (r / 2); e += 32) {
          const int rr = e % rb, a = e / rb;
          const double t0 = Qt[rr + (int64_t)a * rb];
          Qt[rr + (int64_t)a * rb] = Qt[rr + (int64_t)(r - 1 - a) * rb];
          Qt[rr + (int64_t)(r - 1 - a) * rb] = t0;
        }
        __syncwarp();
        warp_upper_solve(rb, Gb, sv, r, Yk, rb);
      }
      __syncthreads();
    } else {
      for (int64_t e = threadIdx.x; e < (int64_t)ra * r; e += blockDim.x) X1[e] = ((e % ra) == (e / ra)) ? 1.0 : 0.0;
      for (int c = threadIdx.x; c < rb; c += blockDim.x) ji[jp[c]] = c;
      __syncthreads();
      cta_apply_q(ra, r, Core, ra, tc, r, X1, (int64_t)ra);
      for (int64_t e = threadIdx.x; e < (int64_t)rb * r; e += blockDim.x) {
        const int c = e % rb, a = e / rb;
        const int row = r - 1 - a, src = ji[c];
        X2[e] = (row <= src) ? Core[row + (int64_t)src * ra] : 0.0;
      }
      __syncthreads();
      cta_householder_qr(rb, r, X2, rb, tc2, red);
      for (int64_t e = threadIdx.x; e < (int64_t)r * r; e += blockDim.x) {
        const int a = e % r, c = e / r;
        const int ra_ = r - 1 - c, ca = r - 1 - a;
        Sw[a + (int64_t)c * A.kcap] = T((ra_ <= ca) ? X2[ra_ + (int64_t)ca * rb] : 0.0);
      }
      for (int64_t e = threadIdx.x; e < (int64_t)rb * r; e += blockDim.x) Qt[e] = ((e % rb) == (e / rb)) ? 1.0 : 0.0;
      __syncthreads();
      cta_apply_q(rb, r, X2, rb, tc2, r, Qt, (int64_t)rb);
      for (int64_t e = threadIdx.x; e < (int64_t)rb * (r / 2); e += blockDim.x) {
        const int rr = e % rb, a = e / rb;
        const double t0 = Qt[rr + (int64_t)a * rb];
        Qt[rr + (int64_t)a * rb] = Qt[rr + (int64_t)(r - 1 - a) * rb];
        Qt[rr + (int64_t)(r - 1 - a) * rb] = t0;
      }
      __syncthreads();
      cta_upper_solve(ra, Ga, su, r, X1, ra);
      cta_upper_solve(rb, Gb, sv, r, Yk, rb);
    }
    // scatter to the stacked order: Xf (su x r) reuses M1, Yf (sv x r) M3
    double* Xf = M1;
    double* Yf = M3;
    for (int64_t e = threadIdx.x; e < (int64_t)su * r; e += blockDim.x) Xf[e] = 0.0;
    __syncthreads();
    for (int64_t e = threadIdx.x; e < (int64_t)ra * r; e += blockDim.x) {
      const int rr = e % ra, c = e / ra;
      Xf[pa[rr] + (int64_t)c * su] = X1[e];
    }
    for (int64_t e = threadIdx.x; e < (int64_t)sv * r; e += blockDim.x) Yf[e] = 0.0;
    __syncthreads();
    for (int64_t e = threadIdx.x; e < (int64_t)rb * r; e += blockDim.x) {
      const int rr = e % rb, c = e / rb;
      Yf[pb[rr] + (int64_t)c * sv] = Yk[e];
    }
    __syncthreads();
    // new bases into temporaries (the target's own U, Vt are operands):
    // U = Uc Xf[:kc] + UL Xf[kc:], V^T = Vc Yf[:kc] + VU Yf[kc:]
    if (r <= 16) {
      cta_gemm_tall(bc, r, kc, Uc, ld, Xf, su, Uo, bc, false);
      cta_gemm_tall(bc, r, p, UL, ld, Xf + kc, su, Uo, bc, true);
      cta_gemm_tall(bk, r, kc, Vc, ld, Yf, sv, Tm, bk, false);
      cta_gemm_tall(bk, r, q, VU, ld, Yf + kc, sv, Tm, bk, true);
    } else {
      cta_gemm<double, GRAM_THREADS>(bc, r, kc, 1.0, Uc, ld, false, Xf, su, false, 0.0, Uo, bc, gsm);
      cta_gemm<double, GRAM_THREADS>(bc, r, p, 1.0, UL, ld, false, Xf + kc, su, false, 1.0, Uo, bc, gsm);
      cta_gemm<double, GRAM_THREADS>(bk, r, kc, 1.0, Vc, ld, false, Yf, sv, false, 0.0, Tm, bk, gsm);
      cta_gemm<double, GRAM_THREADS>(bk, r, q, 1.0, VU, ld, false, Yf + kc, sv, false, 1.0, Tm, bk, gsm);
    }
    T* Uw = A.u(ic, k);
    T* Vw = A.vt(ic, k);
    for (int64_t e = threadIdx.x; e < (int64_t)bc * r; e += blockDim.x) {
      const int rr = e % bc, c = e / bc;
      Uw[rr + (int64_t)c * ld] = T(Uo[e]);
    }
    for (int64_t e = threadIdx.x; e < (int64_t)bk * r; e += blockDim.x) {
      const int rr = e % bk, c = e / bk;
      Vw[rr + (int64_t)c * ld] = T(Tm[e]);
    }
    if (threadIdx.x == 0) A.rank[blk] = r;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Solve kernels.  z is the n x nrhs right-hand side / solution (T, ld n).
// Forward (trsm(L, b, Lower), trsm.cpp:163-174 for a block column B):
//   y_i = Linv_i P_i z_i ; z_j -= L(j,i) y_i for j > i.
// Backward (trsm(U, b, Upper), trsm.cpp:136-145):
//   x_i = Uinv_i z_i ; z_j -= U(j,i) x_i for j < i.
// ---------------------------------------------------------------------------
constexpr int SOLVE_THREADS = 256;
constexpr int SOLVE_ROWS = 16;   // rows of the diagonal solve per CTA
constexpr int SV_NR = 8;         // right-hand sides per pass: one column tile of the FP64 mma
constexpr int SMEM_OPTIN_MAX = 226 * 1024;   // dynamic shared memory a CTA may opt into, beside 1 KB of static

// The solves and the matvec read every factor entry once: memory bounds the
// matvec, the latency of 2 nb dependent steps the solve.  Loads into registers
// left too few bytes in flight (one warp instruction in 17 cycles a scheduler,
// 1.0 TB/s; n = 16384, b = 512, 4 right-hand sides: matvec 452 us, 325 through
// the ring; 8 right-hand sides: refinement 15.1 ms, 7.4 through the ring and 6.3
// with launches that overlap), so a CTA streams its matrices as boxes through a
// ring in shared memory (cp.async, two boxes ahead, also over the seams between
// products) and multiplies them on the tensor pipe with the right-hand sides as
// the columns.  MV_T, MV_T64: out = A^T X, boxes of 256 x 16 and 56 x 64 (rows x
// columns; the second for matrices of few rows: eight outputs a warp and no sum
// over the warps); MV_N*: out = A X, boxes of 512 x 8, 64 x 56 and 16 x 128.  The
// column strides in shared memory make the fragment reads conflict-free.
template <int N> struct IntC { static constexpr int value = N; };
enum : int { MV_T, MV_T64, MV_N512, MV_N64, MV_N16 };
constexpr int MV_BOX = 16 * 260;              // elements of a ring slot (the largest box)

template <typename T>
struct MvSeg {
  const T* A;            // R x C, column stride ld
  int64_t ld;
  int R, C, kind, ldx, ldo, vec;
  const double* X;       // k x nr (shared)
  double* out;           // m x nr (shared); the last segment's results go to the sink
  FRANK_D int m() const { return kind <= MV_T64 ? C : R; }
  FRANK_D int k() const { return kind <= MV_T64 ? R : C; }
  FRANK_D int tm() const { return kind == MV_N512 ? 512 : (kind == MV_N64 || kind == MV_T64 ? 64 : 16); }
  FRANK_D int tk() const { return kind == MV_T ? 256 : (kind == MV_N512 ? 8 : (kind == MV_N16 ? 128 : 56)); }
  FRANK_D void set(const T* A_, int64_t ld_, int R_, int C_, int kind_, const double* X_, int ldx_, double* out_, int ldo_) {
    A = A_; ld = ld_; R = R_; C = C_; kind = kind_; X = X_; ldx = ldx_; out = out_; ldo = ldo_;
    vec = (reinterpret_cast<uintptr_t>(A_) & 15) == 0 && ((ld_ * sizeof(T)) & 15) == 0;
  }
};

// bytes < N: the rest of the N destination bytes is zero-filled
template <int N>
FRANK_D void cp_async(void* dst, const void* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(N), "r"(bytes) : "memory");
}

// Box (r0, c0) of a segment into a slot.  Entries beyond the inner dimension
// are zero-filled (up to the next 16), those beyond the outer one left alone.
template <int BR, int BC, int LDP, bool TR, typename T>
FRANK_D void mv_issue_box(const MvSeg<T>& s, int r0, int c0, T* slot) {
  const int vr = min(BR, s.R - r0), vc = min(BC, s.C - c0);
  const int lr = TR ? min(BR, (vr + 15) & ~15) : vr, lc = TR ? vc : min(BC, (vc + 3) & ~3);
  const T* A = s.A + r0 + (int64_t)c0 * s.ld;
  if (s.vec && vr == BR && vc == BC) {     // a whole box: no predicates, constant strides
    constexpr int E = 16 / (int)sizeof(T), UN = BR / E, CP = UN < SOLVE_THREADS ? SOLVE_THREADS / UN : 1;   // columns per pass
    const int col = threadIdx.x / UN, u = (threadIdx.x % UN) * E;
    const unsigned d = (unsigned)__cvta_generic_to_shared(slot + col * LDP + u);
    const T* src = A + u + (int64_t)col * s.ld;
    const int64_t step = CP * s.ld;
#pragma unroll
    for (int c = 0; c < BC; c += CP)
      if (BC % CP == 0 || c + col < BC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + c * LDP * (int)sizeof(T)), "l"(src) : "memory");
        src += step;
      }
    return;
  }
  auto put = [&](auto e_) {                 // a partial box: the units in use only
    constexpr int E = decltype(e_)::value;
    const int un = (lr + E - 1) / E;
    for (int x = threadIdx.x; x < un * lc; x += SOLVE_THREADS) {
      const int col = x / un, u = (x % un) * E;
      const int ok = col < vc ? max(0, min(E, vr - u)) : 0;
      cp_async<E * (int)sizeof(T)>(slot + col * LDP + u, ok ? A + u + (int64_t)col * s.ld : s.A, ok * (int)sizeof(T));
    }
  };
  if (s.vec) put(IntC<16 / (int)sizeof(T)>{});
  else put(IntC<1>{});
}

// One warp's MI row tiles of a box: k quads q with 4 q < kv, at most KQ of
// them; element (row tile i, quad q) of this lane at a0[i si + q sq].  Every 16
// products start from zero and are added to the sum: 16 + k / 16 roundings
// deep instead of k (the residual of a refinement rests on it).
template <int MI, int KQ, bool FULL, typename T>
FRANK_D void mv_box(const T* a0, int si, int sq, const double* x, int kv, double (&tot)[8][2]) {
  const int t = threadIdx.x & 3;
#pragma unroll
  for (int q0 = 0; q0 < KQ; q0 += 4) {
    if (!FULL && 4 * q0 >= kv) return;
    double acc[MI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i) acc[i][0] = acc[i][1] = 0.0;
#pragma unroll
    for (int q = q0; q < (q0 + 4 < KQ ? q0 + 4 : KQ); ++q) {
      if (!FULL && 4 * q >= kv) break;
      const double xv = FULL || 4 * q + t < kv ? x[4 * q + t] : 0.0;
#pragma unroll
      for (int i = 0; i < MI; ++i) dmma884(acc[i], double(a0[i * si + q * sq]), xv);
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) { tot[i][0] += acc[i][0]; tot[i][1] += acc[i][1]; }
  }
}

template <int MI, int KQ, typename T>
FRANK_D void mv_box(const T* a0, int si, int sq, const double* x, int kv, double (&tot)[8][2]) {
  if (kv >= 4 * KQ) mv_box<MI, KQ, true>(a0, si, sq, x, kv, tot);
  else mv_box<MI, KQ, false>(a0, si, sq, x, kv, tot);
}

// Runs the segments in order; prefetched() is called by all threads once the
// first boxes are on their way (it stages X), sink(row, rhs, value) gets the
// last segment's results, each from one thread.  KINDS: the kinds that occur, a
// bit each (the code of the others costs the short kernels registers and time).
// red: 1024 doubles.
template <int KINDS, typename T, typename Pre, typename Sink>
FRANK_D void mv_run(const MvSeg<T>* seg, int np, int nr, T* ring, int ns, double* red, Pre prefetched, Sink sink) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  auto is = [](int kind, int want) { return ((KINDS >> want) & 1) != 0 && (KINDS == 1 << want || kind == want); };
  int total = 0;
  for (int p = 0; p < np; ++p)
    total += ((seg[p].m() + seg[p].tm() - 1) / seg[p].tm()) * ((seg[p].k() + seg[p].tk() - 1) / seg[p].tk());
  int ip = 0, im = 0, ik = 0, islot = 0, issued = 0;
  auto issue = [&]() {
    if (issued < total) {
      const MvSeg<T>& s = seg[ip];
      T* slot = ring + islot * MV_BOX;
      if (is(s.kind, MV_T)) mv_issue_box<256, 16, 260, true>(s, ik * 256, im * 16, slot);
      else if (is(s.kind, MV_T64)) mv_issue_box<56, 64, 60, true>(s, ik * 56, im * 64, slot);
      else if (is(s.kind, MV_N512)) mv_issue_box<512, 8, 520, false>(s, im * 512, ik * 8, slot);
      else if (is(s.kind, MV_N64)) mv_issue_box<64, 56, 72, false>(s, im * 64, ik * 56, slot);
      else if (is(s.kind, MV_N16)) mv_issue_box<16, 128, 24, false>(s, im * 16, ik * 128, slot);
      ++issued;
      if (++islot == ns) islot = 0;
      if (++ik * s.tk() >= s.k()) {
        ik = 0;
        if (++im * s.tm() >= s.m()) { im = 0; ++ip; }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < ns - 1; ++i) issue();
  prefetched();
  int p = 0, mb = 0, kb = 0, slot_i = 0;
  int cur = -1, kind = 0, m = 0, k = 0, tk = 0, tm = 0;
  const double* X0 = nullptr;
  double tot[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) tot[i][0] = tot[i][1] = 0.0;
  for (int b = 0; b < total; ++b) {
    if (ns == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    issue();
    if (p != cur) {
      const MvSeg<T>& s = seg[p];
      cur = p; kind = s.kind; m = s.m(); k = s.k(); tk = s.tk(); tm = s.tm();
      X0 = s.X + (int64_t)min(g, nr - 1) * s.ldx;
    }
    const T* slot = ring + slot_i * MV_BOX;
    const int m0 = mb * tm, kv = min(tk, k - kb * tk);
    const double* X = X0 + kb * tk;
    if (is(kind, MV_T)) mv_box<2, 8>(slot + g * 260 + wid * 32 + t, 8 * 260, 4, X + wid * 32, kv - wid * 32, tot);
    else if (is(kind, MV_N16)) mv_box<2, 4>(slot + g + (wid * 16 + t) * 24, 8, 96, X + wid * 16, kv - wid * 16, tot);
    else if (is(kind, MV_T64)) {
      if (m0 + wid * 8 < m) mv_box<1, 14>(slot + (wid * 8 + g) * 60 + t, 0, 4, X, kv, tot);
    } else if (is(kind, MV_N64)) {
      if (m0 + wid * 8 < m) mv_box<1, 14>(slot + wid * 8 + g + t * 72, 8, 288, X, kv, tot);
    } else if (is(kind, MV_N512) && m0 + wid * 64 < m) mv_box<8, 2>(slot + wid * 64 + g + t * 520, 8, 2080, X, kv, tot);
    if (++slot_i == ns) slot_i = 0;
    if (++kb * tk < k) continue;
    auto deliver = [&](int row, int c, double v) {
      if (row >= m || c >= nr) return;
      if (p == np - 1) sink(row, c, v);
      else seg[p].out[row + (int64_t)c * seg[p].ldo] = v;
    };
    if (is(kind, MV_T) || is(kind, MV_N16)) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) red[wid * 128 + 8 * i + g + (2 * t + h) * 16] = tot[i][h];
      __syncthreads();
      if (threadIdx.x < 128) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w * 128 + threadIdx.x];
        deliver(m0 + (threadIdx.x & 15), threadIdx.x >> 4, v);
      }
    } else {
      const int per = is(kind, MV_N512) ? 8 : 1;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < per)
#pragma unroll
          for (int h = 0; h < 2; ++h) deliver(m0 + (wid * per + i) * 8 + g, 2 * t + h, tot[i][h]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) tot[i][0] = tot[i][1] = 0.0;
    kb = 0;
    if (++mb * tm >= m) { mb = 0; ++p; }
  }
}

FRANK_HD int sv_ld(int m) { return ((m + 15) & ~15) + 4; }   // = 4 mod 16: conflict-free right-hand-side fragments

// dynamic shared memory of the solve and matvec kernels: the partial tiles,
// x or t2 (bmax x nrhs; kcap <= bmax), t1 (kcap x nrhs) and the ring
template <typename T>
FRANK_HD size_t solve_smem(int bmax, int kcap, int nrhs, int ns) {
  return (1024 + ((size_t)sv_ld(bmax) + sv_ld(kcap)) * nrhs) * sizeof(double) + (size_t)ns * MV_BOX * sizeof(T);
}

// Boxes in the ring: three (two ahead), or two where that lets two CTAs share an SM or fits at all.
template <typename T>
inline int solve_ring(int bmax, int kcap, int nrhs) {
  const size_t two = solve_smem<T>(bmax, kcap, nrhs, 2) + 1024, three = solve_smem<T>(bmax, kcap, nrhs, 3) + 1024;
  const size_t sm = SMEM_OPTIN_MAX + 1024;
  return three > sm || (2 * two <= sm && 2 * three > sm) ? 2 : 3;
}

template <typename T>
struct MvShared {
  double *red, *x, *t1;
  T* ring;
  FRANK_D MvShared(double* p, int bmax, int kcap, int nrhs) {
    red = p;
    x = red + 1024;
    t1 = x + (size_t)sv_ld(bmax) * nrhs;
    ring = reinterpret_cast<T*>(t1 + (size_t)sv_ld(kcap) * nrhs);
  }
};

// A solve is a chain of 4 nb to 6 nb launches of a few microseconds, each launched
// with programmatic stream serialization: its CTAs start, and its ring fetches
// the first boxes (factors, which no launch of the chain writes), while the launch
// before it ends.  Every CTA calls pdl_wait() before it touches vectors, also one
// without work: the end of a grid has to stand for the end of all grids before it.
// (One right-hand side, us a step: b = 512, nb = 32 12.7, with plain launches and
// padded boxes 18.0, 24.9 before the ring; b = 256, nb = 16 9.0, 13.5 and 13.6.)
FRANK_D void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// y = M * P(z_i) (which 0: Linv, permuted input; 1: Uinv),
// y = M^T z_i (2: Uinv^T), or y = P^T (Linv^T z_i) (3), into ybuf (ld bmax).
// grid = ceil(b / SOLVE_ROWS) CTAs, SOLVE_ROWS rows each, from the part of M
// that is not zero.
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS) k_solve_diag(BlrView<T> A, FactorWs<T> ws, int i, const T* z,
                                                              int64_t ldz, int nrhs, int which, T* ybuf, int ns) {
  extern __shared__ __align__(16) double ssm[];
  __shared__ MvSeg<T> seg;
  const int b = A.bs(i), ld = A.bmax, ldx = sv_ld(b);
  const int64_t o = A.off[i];
  const int r0 = blockIdx.x * SOLVE_ROWS, nr = min(SOLVE_ROWS, b - r0);
  if (nr <= 0) { pdl_wait(); return; }
  MvShared<T> sm(ssm, A.bmax, A.kcap, nrhs);
  const T* Mx = (which == 0 || which == 3) ? ws.Linv + (int64_t)i * ld * ld : ws.Uinv + (int64_t)i * ld * ld;
  const int* perm = ws.perm + (int64_t)i * ld;
  const bool lower = which == 0 || which == 2;      // the operator's triangle
  const int k0 = lower ? 0 : r0, k1 = lower ? min(b, r0 + SOLVE_ROWS) : b;
  if (threadIdx.x == 0) {
    if (which <= 1) seg.set(Mx + r0 + (int64_t)k0 * ld, ld, nr, k1 - k0, MV_N16, sm.x, ldx, nullptr, 0);
    else seg.set(Mx + k0 + (int64_t)r0 * ld, ld, k1 - k0, nr, MV_T, sm.x, ldx, nullptr, 0);
  }
  __syncthreads();
  mv_run<1 << MV_N16 | 1 << MV_T>(
      &seg, 1, nrhs, sm.ring, ns, sm.red,
      [&]() {
        pdl_wait();
        for (int r = k0 + threadIdx.x; r < k1; r += SOLVE_THREADS) {
          const T* src = z + o + (which == 0 ? perm[r] : r);
#pragma unroll 8
          for (int c = 0; c < nrhs; ++c) sm.x[r - k0 + c * ldx] = double(src[(int64_t)c * ldz]);
        }
      },
      [&](int r, int c, double v) { ybuf[(which == 3 ? perm[r0 + r] : r0 + r) + (int64_t)c * ld] = T(v); });
}

// Step i's updates z_j -= Blk y_i of every target j, with the solved block y_i
// in ybuf:
// mode 0: targets j > i using blocks (j, i)        [forward, L]
// mode 1: targets j < i using blocks (j, i)        [backward, U]
// mode 2: targets j > i using blocks (i, j)^T      [transpose forward, U^T]
// mode 3: targets j < i using blocks (i, j)^T      [transpose backward, L^T]
// in two launches over all SMs: t1 = inner^T y by 16 columns of the inner
// basis per CTA, then t2 = S t1 and 64 rows of the target per CTA (t2 formed by
// each of them: it is a small part of the reads, and a third launch would cost
// more).  One CTA per target, or a cluster of eight exchanging pieces through
// distributed shared memory, took 41 and 36 us a step at n = 16384, b = 512.
template <typename T>
struct SvTarget {
  int j, bj, gi, gj, r;     // target, its rows, stored block, rank (-1: dense)
  FRANK_D SvTarget(const BlrView<T>& A, int i, int t, int mode) {
    j = (mode == 0 || mode == 2) ? i + 1 + t : t;
    bj = A.bs(j);
    gi = mode >= 2 ? i : j;
    gj = mode >= 2 ? j : i;
    r = A.is_lr(gi, gj) ? A.rank[gi * A.nb + gj] : -1;
  }
};

template <int NT = SOLVE_THREADS, typename T>
FRANK_D void sv_stage(double* x, int ldx, const T* src, int64_t ld, int n, int nrhs) {
  for (int r = threadIdx.x; r < n; r += NT)
#pragma unroll 8
    for (int c = 0; c < nrhs; ++c) x[r + c * ldx] = double(src[r + (int64_t)c * ld]);
}

// grid (ceil(kcap / 16), targets); tbuf: kcap x 8 per target
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS) k_solve_inner(BlrView<T> A, int i, int nrhs, int mode, const T* ybuf,
                                                               double* tbuf, int ns) {
  extern __shared__ __align__(16) double ssm[];
  __shared__ MvSeg<T> seg;
  const SvTarget<T> tg(A, i, blockIdx.y, mode);
  const int c0 = blockIdx.x * 16, ld = A.bmax, bi = A.bs(i), ldx = sv_ld(bi);
  if (c0 >= tg.r) { pdl_wait(); return; }
  MvShared<T> sm(ssm, A.bmax, A.kcap, nrhs);
  if (threadIdx.x == 0)
    seg.set((mode >= 2 ? A.u(tg.gi, tg.gj) : A.vt(tg.gi, tg.gj)) + (int64_t)c0 * ld, ld, bi, min(16, tg.r - c0), MV_T,
            sm.x, ldx, nullptr, 0);
  __syncthreads();
  double* t1 = tbuf + (int64_t)blockIdx.y * A.kcap * SV_NR + c0;
  mv_run<1 << MV_T>(
      &seg, 1, nrhs, sm.ring, ns, sm.red,
      [&]() {
        pdl_wait();
        sv_stage(sm.x, ldx, ybuf, ld, bi, nrhs);
      },
      [&](int r, int c, double v) { t1[r + (int64_t)c * A.kcap] = v; });
}

// grid (ceil(bmax / 64), max(targets, 1)); the first target's CTAs also copy y_i into z_i
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS) k_solve_outer(BlrView<T> A, int i, T* z, int64_t ldz, int nrhs,
                                                               int mode, const T* ybuf, const double* tbuf,
                                                               int ntarget, int ns) {
  extern __shared__ __align__(16) double ssm[];
  __shared__ MvSeg<T> seg[2];
  const int ld = A.bmax, bi = A.bs(i), r0 = blockIdx.x * 64;
  auto wait_and_copy = [&]() {
    pdl_wait();
    if (blockIdx.y == 0)
      for (int r = r0 + (threadIdx.x & 63); r < min(bi, r0 + 64); r += 64)
        for (int c = threadIdx.x >> 6; c < nrhs; c += SOLVE_THREADS / 64)
          z[A.off[i] + r + (int64_t)c * ldz] = ybuf[r + (int64_t)c * ld];
  };
  if ((int)blockIdx.y >= ntarget) { wait_and_copy(); return; }
  const SvTarget<T> tg(A, i, blockIdx.y, mode);
  const bool lr = tg.r >= 0, tr = mode >= 2;
  const int rows = min(64, tg.bj - r0);
  if (rows <= 0 || tg.r == 0) { wait_and_copy(); return; }
  MvShared<T> sm(ssm, A.bmax, A.kcap, nrhs);
  const int k = lr ? tg.r : bi, ldk = sv_ld(k);
  double* x = lr ? sm.t1 : sm.x;
  if (threadIdx.x == 0) {
    if (lr) {
      seg[0].set(A.s(tg.gi, tg.gj), A.kcap, k, k, tr ? MV_T64 : MV_N64, x, ldk, sm.x, ldk);
      seg[1].set((tr ? A.vt(tg.gi, tg.gj) : A.u(tg.gi, tg.gj)) + r0, ld, rows, k, MV_N64, sm.x, ldk, nullptr, 0);
    } else if (tr) {
      seg[0].set(A.dense(tg.gi, tg.gj) + (int64_t)r0 * ld, ld, k, rows, MV_T, x, ldk, nullptr, 0);
    } else {
      seg[0].set(A.dense(tg.gi, tg.gj) + r0, ld, rows, k, MV_N64, x, ldk, nullptr, 0);
    }
  }
  __syncthreads();
  T* zj = z + A.off[tg.j] + r0;
  mv_run<1 << MV_N64 | 1 << MV_T64 | 1 << MV_T>(
      seg, lr ? 2 : 1, nrhs, sm.ring, ns, sm.red,
      [&]() {
        wait_and_copy();
        if (lr) sv_stage(x, ldk, tbuf + (int64_t)blockIdx.y * A.kcap * SV_NR, A.kcap, k, nrhs);
        else sv_stage(x, ldk, ybuf, ld, k, nrhs);
      },
      [&](int r, int c, double v) {
        T* q = zj + r + (int64_t)c * ldz;
        *q = T(double(*q) - v);
      });
}

// Small blocks: one CTA per target does all of a step's update in one launch,
// reading the factors straight into mma fragments.  The chain of a step is then
// too short for a third launch to pay: n = 256 with b = 32, fixed rank 16, four
// right-hand sides 134 us, 147 through the ring; with b = 64 the two are within 10 %
// either way for one to eight right-hand sides; n = 1600 with b = 100 at 1e-3 takes
// 329 us so and 260 through the ring.
constexpr int SD_ROWS = 32;      // rows of the diagonal solve per CTA
FRANK_HD bool solve_direct(int bmax) { return bmax <= 64; }

// One warp's 32 x 8 tile of A X over k0 <= kk < k1: element (i, kk) of A at
// A[i sai + kk sak], X k x nr (shared, ldx); sums as in mv_box.
template <typename T>
FRANK_D void sd_tile(int m, int nr, int k0, int k1, const T* A, int64_t sai, int64_t sak, const double* X, int ldx,
                     int i0, double (&tot)[4][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const T* pa[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pa[i] = A + (int64_t)min(i0 + 8 * i + g, m - 1) * sai + (int64_t)(k0 + t) * sak;
    tot[i][0] = tot[i][1] = 0.0;
  }
  const double* px = X + (int64_t)min(g, nr - 1) * ldx + k0 + t;
  for (int kk = k0; kk < k1; kk += 16) {
    double a[4][4], x[4], acc[4][2];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const bool in = kk + 4 * v + t < k1;
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i][v] = in ? double(pa[i][4 * v * sak]) : 0.0;
      x[v] = in ? px[4 * v] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { pa[i] += 16 * sak; acc[i][0] = acc[i][1] = 0.0; }
    px += 16;
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int i = 0; i < 4; ++i) dmma884(acc[i], a[i][v], x[v]);
#pragma unroll
    for (int i = 0; i < 4; ++i) { tot[i][0] += acc[i][0]; tot[i][1] += acc[i][1]; }
  }
}

// out (m x nr in shared memory, ldo) = A X, X k x nr, by NT threads.  Tiles of 32
// rows; with fewer tiles than warps the inner dimension is cut into slices,
// summed in order.  red: 8 NT doubles.  Ends with a barrier.
template <int NT, typename T>
FRANK_D void sd_mv(int m, int nr, int k, const T* A, int64_t sai, int64_t sak, const double* X, int ldx, double* out,
                   int ldo, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  constexpr int NW = NT / 32;
  const int mt = (m + 31) / 32, sl = max(1, mt >= 5 ? NW / 8 : (mt >= 3 ? NW / 4 : (mt == 2 ? NW / 2 : NW)));
  const int kc = ((k + sl - 1) / sl + 15) & ~15;
  for (int m0 = 0; m0 < mt; m0 += NW / sl) {
    const int tile = m0 + wid / sl, q = wid % sl;
    if (tile < mt) {
      double acc[4][2];
      const int k0 = min(k, q * kc), k1 = min(k, k0 + kc);
      sd_tile(m, nr, k0, k1, A, sai, sak, X, ldx, tile * 32, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) red[wid * 256 + (8 * i + g) + (2 * t + h) * 32] = acc[i][h];
    }
    __syncthreads();
    const int rows = min(m - m0 * 32, (NW / sl) * 32);
    for (int e = threadIdx.x; e < rows * nr; e += NT) {
      const int r = e % rows, c = e / rows;
      double v = 0.0;
      for (int s = 0; s < sl; ++s) v += red[((r >> 5) * sl + s) * 256 + (r & 31) + c * 32];
      out[m0 * 32 + r + c * ldo] = v;
    }
    __syncthreads();
  }
}

// dynamic shared memory: partial tiles, x (bmax), t1 and t2 (kcap; the diagonal solve's SD_ROWS rows) x nrhs
FRANK_HD size_t solve_direct_smem(int bmax, int kcap, int nrhs) {
  return (8 * 256 + ((size_t)sv_ld(bmax) + 2 * (size_t)sv_ld(kcap) + SD_ROWS) * nrhs) * sizeof(double);
}

// k_solve_diag, SD_ROWS rows per CTA
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS) k_solve_diag_direct(BlrView<T> A, FactorWs<T> ws, int i, const T* z,
                                                                     int64_t ldz, int nrhs, int which, T* ybuf) {
  extern __shared__ __align__(16) double ssm[];
  const int b = A.bs(i), ld = A.bmax, ldx = sv_ld(b);
  const int64_t o = A.off[i];
  const int r0 = blockIdx.x * SD_ROWS, nr = min(SD_ROWS, b - r0);
  pdl_wait();
  if (nr <= 0) return;
  double* red = ssm;
  double* out = red + 8 * 256;
  double* x = out + SD_ROWS * nrhs;
  const T* Mx = (which == 0 || which == 3) ? ws.Linv + (int64_t)i * ld * ld : ws.Uinv + (int64_t)i * ld * ld;
  const int* perm = ws.perm + (int64_t)i * ld;
  const bool lower = which == 0 || which == 2;      // the operator's triangle
  const int k0 = lower ? 0 : r0, k1 = lower ? min(b, r0 + SD_ROWS) : b;
  for (int c = threadIdx.x >> 5; c < nrhs; c += SOLVE_THREADS / 32)
    for (int r = k0 + (threadIdx.x & 31); r < k1; r += 32)
      x[r - k0 + c * ldx] = double(z[o + (which == 0 ? perm[r] : r) + (int64_t)c * ldz]);
  __syncthreads();
  if (which <= 1) sd_mv<SOLVE_THREADS>(nr, nrhs, k1 - k0, Mx + r0 + (int64_t)k0 * ld, 1, ld, x, ldx, out, SD_ROWS, red);
  else sd_mv<SOLVE_THREADS>(nr, nrhs, k1 - k0, Mx + k0 + (int64_t)r0 * ld, ld, 1, x, ldx, out, SD_ROWS, red);
  for (int e = threadIdx.x; e < nr * nrhs; e += SOLVE_THREADS) {
    const int r = e % nr, c = e / nr;
    ybuf[(which == 3 ? perm[r0 + r] : r0 + r) + (int64_t)c * ld] = T(out[r + c * SD_ROWS]);
  }
}

// One CTA per target (grid = max(targets, 1)); the first also copies y_i into z_i
template <typename T>
__global__ void __launch_bounds__(SOLVE_THREADS) k_solve_scatter(BlrView<T> A, int i, T* z, int64_t ldz, int nrhs,
                                                                 int mode, const T* ybuf, int ntarget) {
  extern __shared__ __align__(16) double ssm[];
  const int ld = A.bmax, bi = A.bs(i), lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* red = ssm;
  double* ys = red + 8 * 256;
  double* t1 = ys + (size_t)sv_ld(A.bmax) * nrhs;
  double* t2 = t1 + (size_t)sv_ld(A.kcap) * nrhs;
  const int ldy = sv_ld(bi);
  pdl_wait();
  for (int c = wid; c < nrhs; c += SOLVE_THREADS / 32)
    for (int r = lane; r < bi; r += 32) {
      const T v = ybuf[r + (int64_t)c * ld];
      ys[r + c * ldy] = double(v);
      if (blockIdx.x == 0) z[A.off[i] + r + (int64_t)c * ldz] = v;
    }
  if ((int)blockIdx.x >= ntarget) return;
  __syncthreads();
  const SvTarget<T> tg(A, i, blockIdx.x, mode);
  const bool tr = mode >= 2, lr = tg.r >= 0;
  const int r = lr ? tg.r : bi, ldt = lr ? sv_ld(r) : ldy;
  if (lr) {
    const T* S = A.s(tg.gi, tg.gj);
    sd_mv<SOLVE_THREADS>(r, nrhs, bi, tr ? A.u(tg.gi, tg.gj) : A.vt(tg.gi, tg.gj), ld, 1, ys, ldy, t1, ldt, red);
    sd_mv<SOLVE_THREADS>(r, nrhs, r, S, tr ? A.kcap : 1, tr ? 1 : A.kcap, t1, ldt, t2, ldt, red);
  }
  const T* O = lr ? (tr ? A.vt(tg.gi, tg.gj) : A.u(tg.gi, tg.gj)) : A.dense(tg.gi, tg.gj);
  const bool ot = !lr && tr;
  T* zj = z + A.off[tg.j];
  const int g = lane >> 2, q = lane & 3;
  for (int i0 = wid * 32; i0 < tg.bj; i0 += SOLVE_THREADS) {
    double acc[4][2];
    sd_tile(tg.bj, nrhs, 0, r, O, ot ? ld : 1, ot ? 1 : ld, lr ? t2 : ys, ldt, i0, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = i0 + 8 * a + g, c = 2 * q + h;
        if (row < tg.bj && c < nrhs) {
          T* p = zj + row + (int64_t)c * ldz;
          *p = T(double(*p) - acc[a][h]);
        }
      }
  }
}

// ---------------------------------------------------------------------------
// K6: FP64 H-matvec partials: part[(i*nb + j)] = A(i,j) x_j  (bmax x nrhs each),
// or A(j,i)^T x_j when transposing.  One CTA per block, the diagonal's (dense,
// the longest) first; k_matvec_reduce sums over j in fixed order.
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__(SOLVE_THREADS) k_matvec_blocks(BlrView<double> H, const double* x, int64_t ldx,
                                                              int nrhs, double* part, int transpose, int ns) {
  extern __shared__ __align__(16) double ssm[];
  __shared__ MvSeg<double> seg[3];
  const int nb = H.nb, ld = H.bmax, i = blockIdx.x, j = (i + blockIdx.y) % nb;
  const int bi = H.bs(i), bj = H.bs(j), ldb = sv_ld(bj);
  const int gi = transpose ? j : i, gj = transpose ? i : j;   // stored block (gi, gj)
  double* out = part + (int64_t)(i * nb + j) * ld * nrhs;
  const bool lr = H.is_lr(gi, gj), tr = transpose != 0;
  const int r = lr ? H.rank[gi * nb + gj] : 0, ldr = sv_ld(r);
  const int nk = bi > 256 ? MV_N512 : MV_N64;
  if (lr && r == 0) {
    for (int e = threadIdx.x; e < bi * nrhs; e += SOLVE_THREADS) out[e % bi + (int64_t)(e / bi) * ld] = 0.0;
    return;
  }
  MvShared<double> sm(ssm, H.bmax, H.kcap, nrhs);
  if (threadIdx.x == 0) {
    if (lr) {
      seg[0].set(tr ? H.u(gi, gj) : H.vt(gi, gj), ld, bj, r, MV_T, sm.x, ldb, sm.t1, ldr);
      seg[1].set(H.s(gi, gj), H.kcap, r, r, tr ? MV_T : MV_N64, sm.t1, ldr, sm.x, ldr);
      seg[2].set(tr ? H.vt(gi, gj) : H.u(gi, gj), ld, bi, r, nk, sm.x, ldr, nullptr, 0);
    } else if (tr) {
      seg[0].set(H.dense(gi, gj), ld, bj, bi, MV_T, sm.x, ldb, nullptr, 0);
    } else {
      seg[0].set(H.dense(gi, gj), ld, bi, bj, nk, sm.x, ldb, nullptr, 0);
    }
  }
  __syncthreads();
  mv_run<1 << MV_T | 1 << MV_N64 | 1 << MV_N512>(
      seg, lr ? 3 : 1, nrhs, sm.ring, ns, sm.red, [&]() { sv_stage(sm.x, ldb, x + H.off[j], ldx, bj, nrhs); },
      [&](int row, int c, double v) { out[row + (int64_t)c * ld] = v; });
}

// The same without the ring: the CTA reads its block straight into mma fragments
// (sd_mv, sd_tile), and shared memory holds just the vectors (t2 takes x's place),
// so that it does not limit how many CTAs share an SM.  A ring slot is as large
// whatever the block, and its boxes are whole only for blocks of 256 rows and
// more: through the ring alone a product with many small blocks was several waves
// of CTAs waiting at barriers (b = 32, 48 x 48 blocks, one right-hand side 72 us,
// 34 here; b = 128, 32 x 32 55 and 34; b = 512, 8 x 8 100 and 64; one warp per
// column and thread per row, before the ring, 40, 38 and 86).
template <int NT>
static __global__ void __launch_bounds__(NT) k_matvec_direct(BlrView<double> H, const double* x, int64_t ldx, int nrhs,
                                                             double* part, int transpose) {
  extern __shared__ __align__(16) double ssm[];
  const int nb = H.nb, ld = H.bmax, i = blockIdx.x, j = (i + blockIdx.y) % nb;
  const int bi = H.bs(i), bj = H.bs(j), ldb = sv_ld(bj), lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gi = transpose ? j : i, gj = transpose ? i : j;   // stored block (gi, gj)
  double* out = part + (int64_t)(i * nb + j) * ld * nrhs;
  const bool lr = H.is_lr(gi, gj), tr = transpose != 0;
  const int k = lr ? H.rank[gi * nb + gj] : bj, ldk = sv_ld(k);
  if (k == 0) {
    for (int e = threadIdx.x; e < bi * nrhs; e += NT) out[e % bi + (int64_t)(e / bi) * ld] = 0.0;
    return;
  }
  double* red = ssm;
  double* xs = red + 8 * NT;
  double* t1 = xs + (size_t)sv_ld(ld) * nrhs;
  sv_stage<NT>(xs, ldb, x + H.off[j], ldx, bj, nrhs);
  __syncthreads();
  if (lr) {
    const double* S = H.s(gi, gj);
    sd_mv<NT>(k, nrhs, bj, tr ? H.u(gi, gj) : H.vt(gi, gj), ld, 1, xs, ldb, t1, ldk, red);
    sd_mv<NT>(k, nrhs, k, S, tr ? H.kcap : 1, tr ? 1 : H.kcap, t1, ldk, xs, ldk, red);
  }
  const double* O = lr ? (tr ? H.vt(gi, gj) : H.u(gi, gj)) : H.dense(gi, gj);
  const bool ot = !lr && tr;
  const int g = lane >> 2, q = lane & 3;
  for (int i0 = wid * 32; i0 < bi; i0 += NT) {
    double acc[4][2];
    sd_tile(bi, nrhs, 0, k, O, ot ? ld : 1, ot ? 1 : ld, xs, ldk, i0, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = i0 + 8 * a + g, c = 2 * q + h;
        if (row < bi && c < nrhs) out[row + (int64_t)c * ld] = acc[a][h];
      }
  }
}

// Threads of k_matvec_direct, or 0 for the ring: tolerance plans with blocks of
// whole boxes, enough of them to be bound by memory and few right-hand sides (n =
// 16384, b = 512, 3-D at 1e-8: 315 us through the ring and 347 direct for four,
// 380 and 350 for eight; n = 4096 at 1e-6 100 and 64).  128 threads where a block
// has at most four tiles of 32 rows, or five and the grid several waves (b = 128, 48
// x 48 blocks 50 us, 66 with 256 threads; b = 160 74 and 87; b = 256, 24 x 24 at
// 1e-7 131 and 104).
inline int matvec_threads(int bmax, int nb, int nrhs, bool tolerance) {
  if (tolerance && bmax % 512 == 0 && nb >= 16 && nrhs <= 4) return 0;
  return bmax <= 128 || (bmax <= 160 && nb >= 32) ? 128 : 256;
}
FRANK_HD size_t matvec_direct_smem(int bmax, int kcap, int nrhs, int threads) {
  return (8 * (size_t)threads + ((size_t)sv_ld(bmax) + sv_ld(kcap)) * nrhs) * sizeof(double);
}

// y_i = sum_j part(i,j) (fixed order).  If b != null: y = b - A x (residual).
static __global__ void k_matvec_reduce(BlrView<double> H, const double* part, int nrhs, const double* bvec, int64_t ldb,
                                double* y, int64_t ldy) {
  // grid (nb, row tiles of blockDim.x, nrhs)
  const int i = blockIdx.x, h = blockIdx.z;
  const int nb = H.nb, ld = H.bmax;
  const int bi = H.bs(i);
  const int64_t oi = H.off[i];
  const int rr = blockIdx.y * blockDim.x + threadIdx.x;
  if (rr >= bi) return;
  {
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < nb; ++j) s += part[(int64_t)(i * nb + j) * ld * nrhs + rr + (int64_t)h * ld];
    if (bvec) s = bvec[oi + rr + (int64_t)h * ldb] - s;
    y[oi + rr + (int64_t)h * ldy] = s;
  }
}

// column 2-norms squared of an n x nrhs matrix: per-CTA partials part[blk*nrhs + h]
static __global__ void k_colnorm2(const double* v, int64_t n, int64_t ldv, int nrhs, double* part) {
  __shared__ double red[32];
  for (int h = 0; h < nrhs; ++h) {
    double s = 0.0;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
      const double a = v[r + h * ldv];
      s += a * a;
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[blockIdx.x * nrhs + h] = s;
  }
}

template <typename TD, typename TS>
__global__ void k_cast_copy(const TS* src, int64_t lds, TD* dst, int64_t ldd, int64_t n, int nrhs) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * nrhs; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % n, h = e / n;
    dst[r + h * ldd] = TD(src[r + h * lds]);
  }
}

// x += T(d)
// y0 = alpha * y + beta * y0 over n x nrhs (both ld n)
static __global__ void k_axpby(double alpha, const double* y, double beta, double* y0, int64_t n, int nrhs) {
  const int64_t tot = n * nrhs;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x)
    y0[e] = alpha * y[e] + (beta == 0.0 ? 0.0 : beta * y0[e]);
}

template <typename TS>
__global__ void k_axpy_cast(const TS* d, int64_t ldd, double* x, int64_t ldx, int64_t n, int nrhs) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * nrhs; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % n, h = e / n;
    x[r + h * ldx] += double(d[r + h * ldd]);
  }
}

// ---------------------------------------------------------------------------
// Adjoint contraction for the exponential kernel A_ij = exp(-r_ij/theta) +
// nugget*delta_ij: partial sums of sum_h sum_ij lambda_ih (dA_ij/dtheta) x_jh
// with dA/dtheta = exp(-r/theta) r / theta^2, evaluated on the fly (the
// kernel matrix is never formed).  64 x 64 tiles of point pairs per CTA,
// points and vectors staged in shared memory; one partial per CTA, summed on
// the host in a fixed order.
// ---------------------------------------------------------------------------
constexpr int DT_TILE = 64;

static __global__ void __launch_bounds__(256) k_dtheta_contract(const double* x, int dim, int64_t n, double theta,
                                                          const double* lam, int64_t ldl, const double* xv,
                                                          int64_t ldx, int nrhs, double* partial) {
  __shared__ double pi[3][DT_TILE], pj[3][DT_TILE];
  __shared__ double li[8][DT_TILE], xj[8][DT_TILE];
  __shared__ double red[32];
  const int64_t i0 = (int64_t)blockIdx.y * DT_TILE, j0 = (int64_t)blockIdx.x * DT_TILE;
  for (int e = threadIdx.x; e < DT_TILE * dim; e += blockDim.x) {
    const int t = e % DT_TILE, d = e / DT_TILE;
    pi[d][t] = (i0 + t < n) ? x[d * n + i0 + t] : 0.0;
    pj[d][t] = (j0 + t < n) ? x[d * n + j0 + t] : 0.0;
  }
  for (int e = threadIdx.x; e < DT_TILE * nrhs; e += blockDim.x) {
    const int t = e % DT_TILE, h = e / DT_TILE;
    li[h][t] = (i0 + t < n) ? lam[i0 + t + h * ldl] : 0.0;
    xj[h][t] = (j0 + t < n) ? xv[j0 + t + h * ldx] : 0.0;
  }
  __syncthreads();
  double acc = 0.0;
  const double inv_t2 = 1.0 / (theta * theta);
  for (int e = threadIdx.x; e < DT_TILE * DT_TILE; e += blockDim.x) {
    const int a = e % DT_TILE, c = e / DT_TILE;
    if (i0 + a >= n || j0 + c >= n) continue;
    double r2 = 0.0;
    for (int d = 0; d < dim; ++d) { const double t = pi[d][a] - pj[d][c]; r2 += t * t; }
    const double r = sqrt(r2);
    const double da = exp(-r / theta) * r * inv_t2;
    double w = 0.0;
    for (int h = 0; h < nrhs; ++h) w += li[h][a] * xj[h][c];
    acc += da * w;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

// ---------------------------------------------------------------------------
// Construction on the device (FP64): kernel evaluation and compression.
// ---------------------------------------------------------------------------
struct KernelDesc {
  int kind;
  int dim;
  const double* x;   // dim x n, axis-major
  int64_t n;
  double p0, p1;
};

FRANK_D double kernel_eval(const KernelDesc& K, int64_t gi, int64_t gj) {
  double r2 = 0.0;
  for (int d = 0; d < K.dim; ++d) {
    const double t = K.x[d * K.n + gi] - K.x[d * K.n + gj];
    r2 += t * t;
  }
  const double r = sqrt(r2);
  switch (K.kind) {
    case 0: return 1.0 / (r + 1e-3);                                   // functions.cpp:92-109
    case 1: return exp(-1.0 * r2) / (r + 1e-3);                        // functions.cpp:111-128
    case 2: return -log(r + 1e-3) + (gi == gj ? K.p0 : 0.0);
    default: return exp(-r / K.p0) + (gi == gj ? K.p1 : 0.0);
  }
}

// Dense blocks of A_H: one CTA per dense block (listed in blocks[]).
static __global__ void k_build_dense(BlrView<double> H, KernelDesc K, const int* blocks, int nblocks) {
  for (int t = blockIdx.x; t < nblocks; t += gridDim.x) {
    const int blk = blocks[t];
    const int i = blk / H.nb, j = blk % H.nb;
    const int bi = H.bs(i), bj = H.bs(j);
    double* Dm = H.dense(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)bi * bj; e += blockDim.x) {
      const int r = e % bi, c = e / bi;
      Dm[r + (int64_t)c * H.bmax] = kernel_eval(K, H.off[i] + r, H.off[j] + c);
    }
  }
}

// Admissible blocks: evaluate, truncated column-pivoted QR to eps * ||A||_F
// (operations/LAPACK/geqp3.cpp:71-192, LAWN 176 norm down-dating), Q by
// applying the reflectors, R with columns permuted back, then RQ of R
// (via QR of the column-reversed R^T) so S is upper triangular and V has
// orthonormal rows (classes/low_rank.cpp:50-59).  One CTA per block, FP64
// scratch per CTA slot: A (b x b), Q (b x b), X (b x b), norms, pivots.
constexpr int BUILD_THREADS = 512;

static __global__ void __launch_bounds__(BUILD_THREADS) k_build_lowrank(BlrView<double> H, KernelDesc K, const int* blocks,
                                                                 int nblocks, double eps, double* scratch,
                                                                 int64_t stride, int* err) {
  __shared__ double red[32];
  __shared__ int redi[32];
  const int ld = H.bmax;
  double* base = scratch + (int64_t)blockIdx.x * stride;
  double* Am = base;                               // b x b
  double* Qm = Am + (int64_t)ld * ld;              // b x b
  double* Xm = Qm + (int64_t)ld * ld;              // b x b
  double* cnorm = Xm + (int64_t)ld * ld;           // b
  double* partial = cnorm + ld;                    // b
  double* tau = partial + ld;                      // b
  double* tau2 = tau + ld;                         // b
  int* jpvt = reinterpret_cast<int*>(tau2 + ld);   // b
  int* jinv = jpvt + ld;                           // b
  const double dlamch_e = 1.1102230246251565e-16;  // LAPACK dlamch('e') = eps/2 (rounding)
  const double tol3z = sqrt(dlamch_e);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int t = blockIdx.x; t < nblocks; t += gridDim.x) {
    const int blk = blocks[t];
    const int i = blk / H.nb, j = blk % H.nb;
    const int m = H.bs(i), n = H.bs(j);
    const int mind = min(m, n);
    for (int64_t e = threadIdx.x; e < (int64_t)m * n; e += blockDim.x) {
      const int r = e % m, c = e / m;
      Am[r + (int64_t)c * m] = kernel_eval(K, H.off[i] + r, H.off[j] + c);
    }
    __syncthreads();
    double fro = 0.0;
    for (int64_t e = threadIdx.x; e < (int64_t)m * n; e += blockDim.x) fro += Am[e] * Am[e];
    fro = block_sum(fro, red);
    for (int c = wid; c < n; c += nw) {
      double s = 0.0;
      for (int r = lane; r < m; r += 32) s += Am[r + (int64_t)c * m] * Am[r + (int64_t)c * m];
      s = warp_sum(s);
      if (lane == 0) { cnorm[c] = sqrt(s); partial[c] = sqrt(s); jpvt[c] = c; }
    }
    __syncthreads();
    const double threshold = eps * sqrt(fro);
    double maxc;
    {
      double best = -1.0; int bi = -1;
      for (int c = threadIdx.x; c < n; c += blockDim.x) if (cnorm[c] > best) { best = cnorm[c]; bi = c; }
      block_argmax_abs(best < 0 ? 0.0 : best, bi, red, redi, &maxc);
    }
    int r = 0;
    if (maxc <= dlamch_e) {
      // zero block: Q = e_0, R = 0 (geqp3.cpp:97-102)
      for (int e = threadIdx.x; e < m; e += blockDim.x) H.u(i, j)[e] = (e == 0) ? 1.0 : 0.0;
      for (int e = threadIdx.x; e < n; e += blockDim.x) H.vt(i, j)[e] = (e == 0) ? 1.0 : 0.0;
      if (threadIdx.x == 0) { H.s(i, j)[0] = 0.0; H.rank[blk] = 1; }
      __syncthreads();
      continue;
    }
    while (r < mind && maxc > threshold) {
      // pivot: first max over cnorm[r..n)
      double best = -1.0; int bi = -1;
      for (int c = r + threadIdx.x; c < n; c += blockDim.x) if (cnorm[c] > best) { best = cnorm[c]; bi = c; }
      double dummy;
      const int kp = block_argmax_abs(best < 0 ? 0.0 : best, bi, red, redi, &dummy);
      if (kp != r) {
        for (int e = threadIdx.x; e < m; e += blockDim.x) {
          const double a = Am[e + (int64_t)r * m];
          Am[e + (int64_t)r * m] = Am[e + (int64_t)kp * m];
          Am[e + (int64_t)kp * m] = a;
        }
        if (threadIdx.x == 0) {
          double a = cnorm[r]; cnorm[r] = cnorm[kp]; cnorm[kp] = a;
          a = partial[r]; partial[r] = partial[kp]; partial[kp] = a;
          int q = jpvt[r]; jpvt[r] = jpvt[kp]; jpvt[kp] = q;
        }
      }
      __syncthreads();
      // reflector on column r, rows r..m-1 (dlarfg)
      double* col = Am + (int64_t)r * m;
      double s = 0.0;
      for (int e = r + 1 + threadIdx.x; e < m; e += blockDim.x) s += col[e] * col[e];
      const double xn2 = block_sum(s, red);
      const double alpha = col[r];
      double tt = 0.0, beta = alpha, scal = 0.0;
      if (xn2 > 0.0) {
        const double nrm = sqrt(alpha * alpha + xn2);
        beta = alpha >= 0.0 ? -nrm : nrm;
        tt = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
        for (int e = r + 1 + threadIdx.x; e < m; e += blockDim.x) col[e] *= scal;
      }
      __syncthreads();
      if (threadIdx.x == 0) { col[r] = beta; tau[r] = tt; }
      __syncthreads();
      if (r < mind - 1 && tt != 0.0) {
        for (int c = r + 1 + wid; c < n; c += nw) {
          double* cc = Am + (int64_t)c * m;
          double w = (lane == 0) ? cc[r] : 0.0;
          for (int e = r + 1 + lane; e < m; e += 32) w += col[e] * cc[e];
          w = warp_sum(w) * tt;
          if (lane == 0) cc[r] -= w;
          for (int e = r + 1 + lane; e < m; e += 32) cc[e] -= w * col[e];
        }
      }
      __syncthreads();
      // norm down-date (geqp3.cpp:137-159)
      for (int c = r + 1 + wid; c < n; c += nw) {
        if (cnorm[c] != 0.0) {
          double temp = fabs(Am[r + (int64_t)c * m] / cnorm[c]);
          temp = fmax(0.0, (1.0 - temp) * (1.0 + temp));
          const double ratio = cnorm[c] / partial[c];
          const double temp2 = temp * ratio * ratio;
          if (temp2 > tol3z) {
            if (lane == 0) cnorm[c] = cnorm[c] * sqrt(temp);
          } else {
            double s2 = 0.0;
            if (r < m - 1)
              for (int e = r + 1 + lane; e < m; e += 32) s2 += Am[e + (int64_t)c * m] * Am[e + (int64_t)c * m];
            s2 = warp_sum(s2);
            if (lane == 0) { cnorm[c] = (r < m - 1) ? sqrt(s2) : 0.0; partial[c] = cnorm[c]; }
          }
        }
        __syncwarp();
      }
      __syncthreads();
      ++r;
      best = -1.0; bi = -1;
      for (int c = r + threadIdx.x; c < n; c += blockDim.x) if (cnorm[c] > best) { best = cnorm[c]; bi = c; }
      block_argmax_abs(best < 0 ? 0.0 : best, bi, red, redi, &maxc);
      if (r >= n) maxc = 0.0;
    }
    if (r > H.kcap) { if (threadIdx.x == 0) atomicAdd(err + ERR_RANK_OVERFLOW, 1); }
    // Q (m x r) = H_0..H_{r-1} [I_r; 0]
    for (int64_t e = threadIdx.x; e < (int64_t)m * r; e += blockDim.x) {
      const int rr = e % m, c = e / m;
      Qm[rr + (int64_t)c * m] = (rr == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    cta_apply_q(m, r, Am, m, tau, r, Qm, (int64_t)m);
    // inverse pivot: R_perm[:, jpvt[c]] = R[:, c]; build X = (R_perm)^T reversed columns:
    // X (n x r): X[c, a] = R_perm[r-1-a, c]
    for (int c = threadIdx.x; c < n; c += blockDim.x) jinv[jpvt[c]] = c;
    __syncthreads();
    for (int64_t e = threadIdx.x; e < (int64_t)n * r; e += blockDim.x) {
      const int c = e % n, a = e / n;
      const int row = r - 1 - a;
      const int src = jinv[c];
      Xm[c + (int64_t)a * n] = (row <= src) ? Am[row + (int64_t)src * m] : 0.0;
    }
    __syncthreads();
    // QR of X (n x r): X = Qt Rt; S = J Rt^T J, Vt[:, a] = Qt[:, r-1-a]
    cta_householder_qr(n, r, Xm, n, tau2, red);
    const int rs = min(r, H.kcap);
    double* Sd = H.s(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)rs * rs; e += blockDim.x) {
      const int a = e % rs, c = e / rs;
      // S[a][c] = Rt[r-1-c][r-1-a] (upper triangular in (a, c))
      const int ra = r - 1 - c, ca = r - 1 - a;
      Sd[a + (int64_t)c * H.kcap] = (ra <= ca) ? Xm[ra + (int64_t)ca * n] : 0.0;
    }
    // explicit Qt (n x r) into Qm's second half? reuse Am (no longer needed)
    double* Qt = Am;
    for (int64_t e = threadIdx.x; e < (int64_t)n * r; e += blockDim.x) {
      const int rr = e % n, c = e / n;
      Qt[rr + (int64_t)c * n] = (rr == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    cta_apply_q(n, r, Xm, n, tau2, r, Qt, (int64_t)n);
    double* Ud = H.u(i, j);
    double* Vd = H.vt(i, j);
    for (int64_t e = threadIdx.x; e < (int64_t)m * rs; e += blockDim.x) {
      const int rr = e % m, c = e / m;
      Ud[rr + (int64_t)c * ld] = Qm[rr + (int64_t)c * m];
    }
    for (int64_t e = threadIdx.x; e < (int64_t)n * rs; e += blockDim.x) {
      const int rr = e % n, a = e / n;
      Vd[rr + (int64_t)a * ld] = Qt[rr + (int64_t)(r - 1 - a) * n];
    }
    if (threadIdx.x == 0) H.rank[blk] = rs;
    __syncthreads();
  }
}

// Fixed-rank compression of the admissible blocks by randomized SVD
// (classes/low_rank.cpp:40-48 -> operations/randomized/rsvd.cpp:17-29):
// Y = A Omega with the reference's Omega (uniform [0,1), std::mt19937 seeded
// 0, row-major n x p, the same matrix for every block of that width; passed
// in by the host), Q = qr(Y), B = Q^T A, thin SVD of B by one-sided Jacobi
// on B^T with the rotations accumulated in p appended rows, U = Q Ub, then
// truncation to `rank`.  One CTA per block, FP64 scratch slot per CTA:
// A (b x b), Y / Q (b x p), Bt (b + p) x p, small vectors.
static __global__ void __launch_bounds__(BUILD_THREADS) k_build_lowrank_rsvd(BlrView<double> H, KernelDesc K,
                                                                      const int* blocks, int nblocks, int rank,
                                                                      int p, const double* omega_full,
                                                                      const double* omega_last, int64_t stride,
                                                                      double* scratch, int* err) {
  __shared__ double red[32];
  __shared__ double gsm[2 * 16 * 64];
  __shared__ int flag;
  const int ld = H.bmax;
  double* base = scratch + (int64_t)blockIdx.x * stride;
  double* Am = base;                               // m x n
  double* Ym = Am + (int64_t)ld * ld;              // m x p (QR in place)
  double* Qm = Ym + (int64_t)ld * p;               // m x p explicit Q
  double* Bt = Qm + (int64_t)ld * p;               // (n + p) x p
  double* tau = Bt + (int64_t)(ld + p) * p;        // p
  double* sig = tau + p;                           // p
  int* ord = reinterpret_cast<int*>(sig + p);      // p
  for (int t = blockIdx.x; t < nblocks; t += gridDim.x) {
    const int blk = blocks[t];
    const int i = blk / H.nb, j = blk % H.nb;
    const int m = H.bs(i), n = H.bs(j);
    const double* Om = (n == ld) ? omega_full : omega_last;   // n x p row-major
    for (int64_t e = threadIdx.x; e < (int64_t)m * n; e += blockDim.x) {
      const int r = e % m, c = e / m;
      Am[r + (int64_t)c * m] = kernel_eval(K, H.off[i] + r, H.off[j] + c);
    }
    __syncthreads();
    // Y = A Omega: Omega row-major n x p == column-major p x n, used transposed
    cta_gemm<double, BUILD_THREADS>(m, p, n, 1.0, Am, m, false, Om, p, true, 0.0, Ym, m, gsm);
    cta_householder_qr(m, p, Ym, m, tau, red);
    for (int64_t e = threadIdx.x; e < (int64_t)m * p; e += blockDim.x) {
      const int r = e % m, c = e / m;
      Qm[e] = (r == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    cta_apply_q(m, p, Ym, m, tau, p, Qm, (int64_t)m);
    // Bt (n x p) = (Q^T A)^T = A^T Q; identity appended below (p x p)
    cta_gemm<double, BUILD_THREADS>(n, p, m, 1.0, Am, m, true, Qm, m, false, 0.0, Bt, n + p, gsm);
    for (int e = threadIdx.x; e < p * p; e += blockDim.x) {
      const int r = e % p, c = e / p;
      Bt[(n + r) + (int64_t)c * (n + p)] = (r == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    const int sweeps = cta_jacobi_columns(n, p, Bt, n + p, 60, &flag, n + p);
    if (sweeps < 0 && threadIdx.x == 0) atomicAdd(err + ERR_JACOBI, 1);
    // Bt columns: W Sigma (top n rows), Z (bottom p rows); B = Z Sigma W^T
    for (int c = threadIdx.x >> 5; c < p; c += blockDim.x >> 5) {
      double sacc = 0.0;
      for (int r = threadIdx.x & 31; r < n; r += 32) sacc += Bt[r + (int64_t)c * (n + p)] * Bt[r + (int64_t)c * (n + p)];
      sacc = warp_sum(sacc);
      if ((threadIdx.x & 31) == 0) sig[c] = sqrt(sacc);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < p; c += blockDim.x) {
      const double v = sig[c];
      int pos = 0;
      for (int d = 0; d < p; ++d) pos += sorts_before(sig[d], d, v, c);
      ord[pos] = c;
    }
    __syncthreads();
    const int rk = min(rank, H.kcap);
    if (rank > H.kcap && threadIdx.x == 0) atomicAdd(err + ERR_RANK_OVERFLOW, 1);
    double* Ud = H.u(i, j);
    double* Vd = H.vt(i, j);
    double* Sd = H.s(i, j);
    // U = Q Z[:, ord] (m x rk); Vt = W[:, ord] (n x rk) normalised; S = diag
    for (int64_t e = threadIdx.x; e < (int64_t)m * rk; e += blockDim.x) {
      const int r = e % m, c = e / m;
      const int src = ord[c];
      double acc = 0.0;
      for (int t = 0; t < p; ++t) acc += Qm[r + (int64_t)t * m] * Bt[(n + t) + (int64_t)src * (n + p)];
      Ud[r + (int64_t)c * ld] = acc;
    }
    for (int64_t e = threadIdx.x; e < (int64_t)n * rk; e += blockDim.x) {
      const int r = e % n, c = e / n;
      const int src = ord[c];
      const double sv = sig[src];
      Vd[r + (int64_t)c * ld] = sv > 0.0 ? Bt[r + (int64_t)src * (n + p)] / sv : 0.0;
    }
    for (int64_t e = threadIdx.x; e < (int64_t)rk * rk; e += blockDim.x) {
      const int r = e % rk, c = e / rk;
      Sd[r + (int64_t)c * H.kcap] = (r == c) ? sig[ord[c]] : 0.0;
    }
    if (threadIdx.x == 0) H.rank[blk] = rk;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Batched factorization of independent systems: one launch per elimination
// step covers every system of a batch (grid.z = system).  Each CTA reads its
// system's views and parameters from a device table and leaves at once when
// its system has no step i or fewer tasks than its block index; the bodies
// are the single-system kernels' own.
// ---------------------------------------------------------------------------
template <typename T>
struct SysDev {
  BlrView<double> H;
  BlrView<T> W;
  FactorWs<T> ws;
  int* work;              // recompression task counters of the system ([nb])
  double* rscratch;       // reset-truncation scratch (k_truncate_lr)
  int64_t rstride;
  double core_scale, thr_trunc;
  int smax, core_method, proj_tol, split_p, core_smem, dupd_band, pretrunc, has_lr;
};

template <typename T>
__global__ void k_reset_b(const SysDev<T>* S) {
  const SysDev<T>& s = S[blockIdx.z];
  if ((int)blockIdx.x >= s.H.nb * s.H.nb) return;
  k_reset_impl<T>(s.H, s.W);
}

template <typename T>
__global__ void __launch_bounds__(TRUNC_THREADS) k_truncate_lr_b(const SysDev<T>* S) {
  const SysDev<T>& s = S[blockIdx.z];
  if (!s.pretrunc) return;
  k_truncate_lr_impl<T>(s.H, s.W, s.ws, s.thr_trunc, s.rscratch, s.rstride);
}

template <typename T>
__global__ void __launch_bounds__(LEAF_THREADS) k_leaf_step_b(const SysDev<T>* S, int i, int p) {
  const SysDev<T>& s = S[blockIdx.z];
  if (i >= s.W.nb) return;
  k_leaf_step_impl<T>(s.W, s.ws, i, p);
}

template <typename T>
__global__ void __launch_bounds__(LEAF_THREADS) k_leaf_final_b(const SysDev<T>* S, int i) {
  const SysDev<T>& s = S[blockIdx.z];
  if (i >= s.W.nb) return;
  k_leaf_final_impl<T>(s.W, s.ws, i);
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_gather_b(const SysDev<T>* S, int i) {
  const SysDev<T>& s = S[blockIdx.z];
  if ((int)blockIdx.x >= s.W.nb - i - 1) return;
  k_panel_gather_impl<T>(s.W, s.ws, i);
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_mul_b(const SysDev<T>* S, int i) {
  const SysDev<T>& s = S[blockIdx.z];
  if ((int)blockIdx.x >= 2 * (s.W.nb - i - 1)) return;
  k_panel_mul_impl<T>(s.W, s.ws, i);
}

template <typename T>
__global__ void __launch_bounds__(PANEL_THREADS) k_panel_fin_b(const SysDev<T>* S, int i) {
  const SysDev<T>& s = S[blockIdx.z];
  if ((int)blockIdx.x >= 2 * (s.W.nb - i - 1)) return;
  k_panel_fin_impl<T>(s.W, s.ws, i);
}

template <typename T>
__global__ void __launch_bounds__(DUPD_THREADS) k_update_dense_b(const SysDev<T>* S, int i, int mode) {
  const SysDev<T>& s = S[blockIdx.z];
  if (i >= s.W.nb - 1) return;
  k_update_dense_impl<T>(s.W, s.ws, i, s.dupd_band, mode);
}

template <typename T>
__global__ void __launch_bounds__(RECOMP_THREADS) k_recompress_b(const SysDev<T>* S, int i) {
  const SysDev<T>& s = S[blockIdx.z];
  if (i >= s.W.nb - 1 || !s.has_lr) return;
  // the views in shared memory (as kernel parameters would be in constant memory)
  __shared__ BlrView<T> A;
  __shared__ FactorWs<T> ws;
  if (threadIdx.x == 0) { A = s.W; ws = s.ws; }
  __syncthreads();
  k_recompress_impl<T>(A, ws, i, s.smax, s.core_method, s.core_scale, 0, s.work + i, 0, nullptr, nullptr,
                       s.proj_tol, s.split_p, s.core_smem);
}

}  // namespace frank
