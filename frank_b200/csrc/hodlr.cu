// Multi-level H-LU on the device: FRANK's recursive getrf_omm(Hierarchical)
// (operations/LAPACK/getrf.cpp:45-65) for a Hierarchical matrix with a binary
// cluster tree and weak admissibility -- Hierarchical(kernel, params, n, n,
// rank, nleaf, admis = 0, 2, 2) (classes/hierarchical.cpp:49-109,
// matrix_initializer.cpp:51-58 position-based: every off-diagonal child is
// LowRank, every diagonal child recurses until it is a dense leaf), fixed
// rank k.
//
// Layout in HBM (FP64, column-major), levels l = 1 .. L, n = b 2^L:
//   leaves      D[p]        b x b, p = 0 .. 2^L - 1 (A_H: D0; factor: D,
//                            packed pivoted LU after getrf)
//   LowRank     (l, c)      c = 0 .. 2^l - 1: rows of cluster c of level l,
//                            columns of its sibling c ^ 1, size s_l = n >> l:
//                            U (s_l x k), S (k x k), V (k x s_l, ld k); all
//                            blocks of a level are one contiguous slab, so a
//                            level's blocks are one strided batch
//   per leaf    Linv, Uinv, Uinv^T (b x b), pivots.
//
// getrf(node) = getrf(left); U_up <- L_left^{-1} P U_up and V_low <- V_low
// U_left^{-1} (level-parallel substitutions on the left subtree, see
// enqueue_sub); the Schur update
// -L_low U_up = LowRank(U_low, S', V_up), S' = -(S_low V_low)(U_up S_up)
// (gemm.cpp:374-393), added into the right child by splitting it over the
// child's blocks (addition.cpp:62-66): dense leaves += (U S') V, LowRank
// blocks += by the batched LowRank addition of ops.cu (fast_rounded_addition,
// the reference's default for fixed rank, addition.cpp:133-203, or
// rounded_addition), one launch per level and parity; then getrf(right).
// The shapes are static (fixed rank), so the whole factorization is one
// stream of launches, captured once into a CUDA graph and replayed.
//
// Pivoting: the leaves take dgetrf's partial pivoting with the interchanges
// applied (P A = L U with P = blockdiag(P_p)); the L blocks keep their rows
// in natural order and each substitution applies P_p with leaf p's inverse,
// which is the same thing.  The
// reference discards the pivots (getrf.cpp:67-84); the two agree whenever
// dgetrf does not swap rows.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#include <algorithm>

// The BLR engine's kernels (leaf LU, explicit inverses, kernel evaluation)
// are compiled into this translation unit under a private name, so that none
// of their symbols collides with the engine's own copy in api.cu.
#define frank frank_blr_private
namespace {
#include "blr_kernels.cuh"
namespace blr = frank_blr_private;
}  // namespace
#undef frank

#include "../../include/frank_b200.h"
#include "ops_tasks.h"

#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace frank {
int set_error(int code, const std::string& msg);
namespace ops {
int64_t qr_ws(int m, int n);
int64_t svd_scratch(int m, int n);
int64_t lr_add_ws(int m, int n, int ka, int kb);
void launch_gemm(cudaStream_t s, int m, int n, int k, int count, double alpha, const double* a, int64_t lda,
                 int64_t sa, bool ta, const double* b, int64_t ldb, int64_t sb, bool tb, double beta, double* c,
                 int64_t ldc, int64_t sc);
void launch_qr(cudaStream_t s, int m, int n, int count, const double* a, int64_t lda, int64_t sa, double* q,
               int64_t ldq, int64_t sq, double* r, int64_t ldr, int64_t sr, double* scratch, int64_t ws);
void launch_svd(cudaStream_t s, int m, int n, int count, const double* a, int64_t lda, int64_t sa, double* u,
                int64_t ldu, int64_t su, double* sv, int64_t ss, double* vt, int64_t ldvt, int64_t svt,
                double* scratch, int64_t ws, int* err);
int lr_add_prepare();
void launch_lr_add_tasks(cudaStream_t s, int count, int mmax, const LrAddTask* tasks, int kmax, int fast,
                         double* scratch, int* err);
}  // namespace ops
}  // namespace frank

namespace {
namespace hk {

using blr::KernelDesc;
using blr::kernel_eval;

constexpr int HMAX_RANK = 64;   // largest accepted rank
constexpr int HMAX_LEAF = 512;  // b <= 512
constexpr int WT = 256;         // threads of the update / matvec kernels
constexpr int KG_P = 72;        // rsvd sample width the construction product holds (k + 5 <= 69)

enum { HERR_JACOBI = 8, HERR_RANK = 9, HERR_SLOTS = 16 };

// Device view of one H-matrix's blocks (working copy or A_H).
struct HView {
  int64_t n;
  int b, L, k;
  const double* D;
  const double* U;
  const double* S;
  const double* V;
  FRANK_D int64_t s(int l) const { return n >> l; }
  FRANK_D const double* u(int l, int c) const { return U + (int64_t)(l - 1) * n * k + (int64_t)c * s(l) * k; }
  FRANK_D const double* v(int l, int c) const { return V + (int64_t)(l - 1) * n * k + (int64_t)c * s(l) * k; }
  FRANK_D const double* sm(int l, int c) const { return S + ((int64_t)(1 << l) - 2 + c) * k * k; }
};

struct LeafFactors {
  const double* Linv;   // [P][b*b] unit lower inverse
  const double* Uinv;   // [P][b*b] upper inverse
  const double* UinvT;  // [P][b*b] transpose of Uinv (lower)
  const int* perm;      // [P][b] (P_p r)[i] = r[perm[i]]
};

// ---------------------------------------------------------------------------
// Level-parallel substitution on a subtree (node (l0, c0) and everything below
// it).  With W = M_right(U_low), Z = U_left^{-1} U_up and Zt = U_right^{-T}
// V_up^T precomputed per node (M the pivoted forward substitution), the three
// substitutions are: every leaf at once, then for each level from the bottom
// up, every node at once:
//   mode 0  X <- L^{-1} P X : x_right -= W  S_low  (V_low  x_left)
//   mode 1  X <- U^{-T} X   : x_right -= Zt S_up^T (U_up^T x_left)
//   mode 2  X <- U^{-1} X   : x_left  -= Z  S_up   (V_up   x_right)
// (from L = [[L_l, 0], [U S V, L_r]] and U likewise), and the H-matvec has the
// same two kernels per level:
//   mode 3  Y = A X         : y(rows of c) += U_c S_c (V_c x(rows of c ^ 1)).
// The walks over the leaves that did modes 0 to 2 before kept eight CTAs busy
// with a chain of 2^h leaf steps (8.9 ms for the top of an n = 32768 tree).
// The columns of X (right-hand sides, or the k columns of a basis) go through
// the FP64 tensor pipe 32 at a time, so a block is read once for all of them.
// ---------------------------------------------------------------------------
struct HJob {
  int mode;
  const double* src;      // leaves read X here: element (i, c) at src[i srs + c scs]
  int64_t srs, scs;
  double* X;              // result, and X of the level steps: X[i xrs + c ldx] (xrs = 1 above the leaves)
  int64_t xrs, ldx;
  const double* xin;      // mode 3: the vector multiplied (X is the result)
  int64_t ldin;
};

constexpr int HC = 32;            // columns of X per CTA
constexpr int HLC = 8;            // columns per CTA of the leaf step
constexpr int HPASS = 128;        // columns of a solve or product per pass: bounds its buffers
constexpr int H_CHUNK = 512;      // least rows per partial product
constexpr int H_NCH = 64;         // most partial products of one block
constexpr int H_TSMEM = 8 * HC * HC * 8;   // dynamic shared memory of the partial products

// Rows of a block of order s per partial product, and their number.
inline __host__ __device__ int64_t h_chunk(int64_t s) {
  const int64_t c = (s + H_NCH - 1) / H_NCH;
  return c < H_CHUNK ? (int64_t)H_CHUNK : c;
}
inline __host__ __device__ int h_nch(int64_t s) { return (int)((s + h_chunk(s) - 1) / h_chunk(s)); }

// X_p <- Op_p X_p for the leaves p0 .. of a subtree (Linv P, Uinv^T, Uinv or the
// leaf of A_H itself); grid (leaves, groups of HLC columns, jobs).
__global__ void __launch_bounds__(WT) k_h_leaf_mm(HView h, LeafFactors f, HJob j0, HJob j1, int p0, int ncols) {
  __shared__ double R[HLC * (HMAX_LEAF + 4)];
  const HJob& J = blockIdx.z ? j1 : j0;
  const int p = p0 + blockIdx.x, b = h.b, c0 = blockIdx.y * HLC, nc = min(HLC, ncols - c0);
  const int64_t r0 = (int64_t)blockIdx.x * b;
  const int ldr = ((b + 15) & ~15) + 4;
  const int* perm = f.perm + (int64_t)p * b;
  for (int e = threadIdx.x; e < nc * b; e += WT) {
    const int i = J.srs == 1 ? e % b : e / nc, c = J.srs == 1 ? e / b : e % nc;
    R[i + c * ldr] = J.src[(r0 + (J.mode == 0 ? perm[i] : i)) * J.srs + (c0 + c) * J.scs];
  }
  __syncthreads();
  const double* Op = (J.mode == 0 ? f.Linv : J.mode == 1 ? f.UinvT : J.mode == 2 ? f.Uinv : h.D) + (int64_t)p * b * b;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int i0 = (threadIdx.x >> 5) * 32; i0 < b; i0 += WT) {
    double acc[4][1][2];
    // the operators of modes 0 and 1 are lower triangular, that of mode 2 upper
    const int k0 = J.mode == 2 ? i0 : 0, k1 = J.mode <= 1 ? min(b, i0 + 32) : b;
    blr::warp_dgemm_acc<4, 1, false>(b, nc, k0, k1, Op, 1, b, R, ldr, 1, i0, 0, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = i0 + 8 * i + g, c = 2 * t + q;
        if (r < b && c < nc) J.X[(r0 + r) * J.xrs + (c0 + c) * J.ldx] = acc[i][0][q];
      }
  }
}

// One CTA's share of T (m <= HC, n <= 8 NJ <= HC) = A B over rows [k0, k1), element (i,
// kk) of A at A[i sai + kk sak], B col-major: eight warps take an eighth of the rows
// each and sum in shared memory (red, 8 HC HC doubles); sink(i, j, value) gets the
// results, each from one thread.  NJ = 1 for up to eight columns: n = 512 in leaves of
// 32, one right-hand side, takes 93 us a solve so and 108 with the products and sums
// of 32 columns (106 by the walks before).
template <int NJ, typename Sink>
__device__ __forceinline__ void h_tprod(int m, int n, int64_t k0, int64_t k1, const double* A, int64_t sai, int64_t sak,
                                        const double* B, int64_t ldb, double* red, Sink sink) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, wid = threadIdx.x >> 5;
  const int64_t len = ((k1 - k0 + 7) / 8 + 3) & ~(int64_t)3;
  const int64_t a0 = min(k1, k0 + wid * len), a1 = min(k1, a0 + len);
  double acc[4][NJ][2];
  blr::warp_dgemm_acc<4, NJ, false>(m, n, 0, (int)(a1 - a0), A + a0 * sak, sai, sak, B + a0, ldb, 1, 0, 0, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) red[wid * HC * 8 * NJ + (8 * i + g) + (8 * j + 2 * t + q) * HC] = acc[i][j][q];
  __syncthreads();
#pragma unroll
  for (int x = 0; x < HC * 8 * NJ / WT; ++x) {
    const int e = threadIdx.x + x * WT;
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += red[w * HC * 8 * NJ + e];
    if (e % HC < m && e / HC < n) sink(e % HC, e / HC, v);
  }
  __syncthreads();
}

// T2 (k x ncols per node, ld k) = op(S) (inner product of the block with its side of
// X) for the nodes of one level of a subtree: grid (chunks, nodes, jobs x column
// groups).  The chunk that finishes last sums all of them in order and applies S.
__global__ void __launch_bounds__(WT) k_h_t(HView h, HJob j0, HJob j1, int njobs, int l, int first, int ncols,
                                            double* part, double* T2, int* counter) {
  extern __shared__ double red[];
  __shared__ double t1[HMAX_RANK * HC];
  __shared__ int last;
  const int job = blockIdx.z % njobs, grp = blockIdx.z / njobs;
  const HJob& J = job ? j1 : j0;
  const int k = h.k, nc = min(HC, ncols - grp * HC), nch = gridDim.x, node = blockIdx.y;
  const int64_t sl = h.s(l), chunk = h_chunk(sl), i0 = blockIdx.x * chunk, i1 = min(sl, i0 + chunk);
  // the block, and the cluster whose rows of X it reads
  const int c = J.mode == 3 ? node : (J.mode == 0 ? first + 2 * node + 1 : first + 2 * node);
  const int xc = J.mode == 0 || J.mode == 1 ? first + 2 * node : (J.mode == 2 ? first + 2 * node + 1 : c ^ 1);
  const bool tr = J.mode == 1;
  const double* A = tr ? h.u(l, c) : h.v(l, c);
  const double* x = (J.mode == 3 ? J.xin : J.X) + (int64_t)(xc - (J.mode == 3 ? 0 : first)) * sl;
  const int64_t ldx = J.mode == 3 ? J.ldin : J.ldx;
  x += (int64_t)grp * HC * ldx;
  const int64_t slot = ((int64_t)blockIdx.z * gridDim.y + node);
  double* pt = part + slot * nch * k * HC;
  for (int m0 = 0; m0 < k; m0 += HC) {
    const int m = min(HC, k - m0);
    auto keep = [&](int r, int q, double v) {
      if (nch == 1) t1[m0 + r + q * k] = v;
      else pt[(int64_t)blockIdx.x * k * HC + m0 + r + q * k] = v;
    };
    const double* Am = A + (tr ? (int64_t)m0 * sl : m0);
    if (nc <= 8) h_tprod<1>(m, nc, i0, i1, Am, tr ? sl : 1, tr ? 1 : k, x, ldx, red, keep);
    else h_tprod<4>(m, nc, i0, i1, Am, tr ? sl : 1, tr ? 1 : k, x, ldx, red, keep);
  }
  if (nch > 1) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      last = atomicAdd(counter + slot, 1) == nch - 1;
      if (last) counter[slot] = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int e = threadIdx.x; e < k * nc; e += WT) {
      double v = 0.0;
#pragma unroll 8
      for (int q = 0; q < nch; ++q) v += pt[(int64_t)q * k * HC + e];
      t1[e] = v;
    }
    __syncthreads();
  }
  const double* S = h.sm(l, c);
  double* out = T2 + ((int64_t)(job * gridDim.y + node) * ncols + grp * HC) * k;
  for (int e = threadIdx.x; e < k * nc; e += WT) {
    const int r = e % k, q = e / k;
    double v = 0.0;
#pragma unroll 4
    for (int t = 0; t < k; ++t) v = fma(tr ? S[t + r * k] : S[r + t * k], t1[t + q * k], v);
    out[e] = v;
  }
}

// X(rows of the node's target) -= outer T2 (mode 3: +=); outer from the slabs W (modes
// 0, 2), Zt (mode 1) or the block's own U; grid (row tiles of WT, nodes, jobs x
// column groups).
__global__ void __launch_bounds__(WT) k_h_u(HView h, const double* WZ, const double* WT_, HJob j0, HJob j1, int njobs,
                                            int l, int first, int ncols, const double* T2) {
  __shared__ double ts[HC * (HMAX_RANK + 4)];
  const int job = blockIdx.z % njobs, grp = blockIdx.z / njobs, node = blockIdx.y;
  const HJob& J = job ? j1 : j0;
  const int k = h.k, nc = min(HC, ncols - grp * HC);
  const int64_t sl = h.s(l), r0 = (int64_t)blockIdx.x * WT;
  const int rows = (int)min((int64_t)WT, sl - r0);
  const int c = J.mode == 3 ? node : (J.mode == 0 ? first + 2 * node + 1 : first + 2 * node);
  const int target = J.mode == 1 ? c + 1 : c;       // cluster whose rows are updated
  const int64_t off = (int64_t)(l - 1) * h.n * k + (int64_t)c * sl * k;
  const double* O = (J.mode == 3 ? h.U : J.mode == 1 ? WT_ : WZ) + off + r0;
  const int ldt = ((k + 15) & ~15) + 4;
  const double* t2 = T2 + ((int64_t)(job * gridDim.y + node) * ncols + grp * HC) * k;
  for (int e = threadIdx.x; e < k * nc; e += WT) ts[e % k + (e / k) * ldt] = t2[e];
  __syncthreads();
  double* X = J.X + (int64_t)(target - (J.mode == 3 ? 0 : first)) * sl + r0 + (int64_t)grp * HC * J.ldx;
  blr::warps_dgemm<4, 2>(threadIdx.x >> 5, WT / 32, rows, nc, k, J.mode == 3 ? 1.0 : -1.0, O, 1, sl, ts, ldt, 1, 1.0, X,
                         J.ldx);
}

// A (k x s, ld k) = X^T (s x k, ld s).
__global__ void __launch_bounds__(WT) k_h_transpose(int64_t s, int k, const double* X, double* A) {
  __shared__ double t[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int c0 = blockIdx.y * 32, lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  for (int c = ly; c < 32; c += WT / 32)
    if (i0 + lx < s && c0 + c < k) t[c][lx] = X[i0 + lx + (int64_t)(c0 + c) * s];
  __syncthreads();
  for (int i = ly; i < 32; i += WT / 32)
    if (i0 + i < s && c0 + lx < k) A[c0 + lx + (i0 + i) * k] = t[lx][i];
}

// S' = -(S_low (V_low U_up) S_up) (k x k) for the Schur update of a node:
// V_low (k x s, ld k), U_up (s x k, ld s).  A CTA per chunk of s; the last one to
// finish (counter, which returns to 0) sums the chunks in order and forms S'.
__global__ void __launch_bounds__(WT) k_h_core(int64_t s, int k, const double* Vl, const double* Uu, const double* Sl,
                                               const double* Su, double* part, double* Sp, int* counter) {
  extern __shared__ double red[];                 // 8 HC HC; then X and Y (k x k each)
  __shared__ int last;
  const int64_t chunk = h_chunk(s), i0 = blockIdx.x * chunk, i1 = min(s, i0 + chunk);
  const int kk = k * k;
  double* mine = part + (int64_t)blockIdx.x * kk;
  for (int m0 = 0; m0 < k; m0 += HC)
    for (int n0 = 0; n0 < k; n0 += HC) {
      const int m = min(HC, k - m0), n = min(HC, k - n0);
      h_tprod<4>(m, n, i0, i1, Vl + m0, 1, k, Uu + (int64_t)n0 * s, s, red,
                 [&](int r, int q, double v) { mine[m0 + r + (n0 + q) * k] = v; });
    }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
    if (last) *counter = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double* X = red;
  double* Y = red + kk;
  for (int e = threadIdx.x; e < kk; e += WT) {
    double v = 0.0;
#pragma unroll 8
    for (int q = 0; q < (int)gridDim.x; ++q) v += part[(int64_t)q * kk + e];
    X[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kk; e += WT) {    // Y = S_low X
    double v = 0.0;
#pragma unroll 4
    for (int q = 0; q < k; ++q) v = fma(Sl[e % k + q * k], X[q + (e / k) * k], v);
    Y[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kk; e += WT) {    // S' = -(Y S_up)
    double v = 0.0;
#pragma unroll 4
    for (int q = 0; q < k; ++q) v = fma(Y[e % k + q * k], Su[q + (e / k) * k], v);
    Sp[e] = -v;
  }
}

// Dense leaves of A_H: D[p] = K(rows of p, cols of p).
__global__ void k_h_build_leaves(KernelDesc K, int b, int P, double* D) {
  const int64_t tot = (int64_t)P * b * b;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = e / ((int64_t)b * b);
    const int r = (int)(e % b), c = (int)((e / b) % b);
    D[e] = kernel_eval(K, p * b + r, p * b + c);
  }
}

// Z (s x p) = K(R, C) W for every block c of a level (blockIdx.y): R the
// rows of cluster c, C the rows of its sibling (swap = 0), or the two
// exchanged (swap = 1, the transposed product K(C, R) of an off-diagonal
// block, used for Q^T A).  The kernel is evaluated tile by tile, never
// stored.  W, Z: ld s, block stride s p.
__global__ void __launch_bounds__(WT) k_h_kgemm(KernelDesc K, int64_t s, int p, int swap, const double* W,
                                                double* Z) {
  __shared__ double Ks[64][33];
  __shared__ double Ws[32][KG_P];
  const int c = blockIdx.y;
  const int64_t R0 = (int64_t)(swap ? (c ^ 1) : c) * s, C0 = (int64_t)(swap ? c : (c ^ 1)) * s;
  const double* Wc = W + (int64_t)c * s * p;
  double* Zc = Z + (int64_t)c * s * p;
  const int64_t r0 = (int64_t)blockIdx.x * 64;
  const int tid = threadIdx.x, row = tid & 63, g = tid >> 6;
  const int rn = (int)min((int64_t)64, s - r0);
  double acc[KG_P / 4];
#pragma unroll
  for (int u = 0; u < KG_P / 4; ++u) acc[u] = 0.0;
  for (int64_t t0 = 0; t0 < s; t0 += 32) {
    const int tn = (int)min((int64_t)32, s - t0);
    for (int e = tid; e < 64 * 32; e += WT) {
      const int i = e % 64, t = e / 64;
      Ks[i][t] = (i < rn && t < tn) ? kernel_eval(K, R0 + r0 + i, C0 + t0 + t) : 0.0;
    }
    for (int e = tid; e < 32 * p; e += WT) {
      const int t = e % 32, j = e / 32;
      Ws[t][j] = t < tn ? Wc[(t0 + t) + (int64_t)j * s] : 0.0;
    }
    __syncthreads();
    for (int t = 0; t < 32; ++t) {
      const double kv = Ks[row][t];
#pragma unroll
      for (int u = 0; u < KG_P / 4; ++u) {
        const int j = g + 4 * u;
        if (j < p) acc[u] += kv * Ws[t][j];
      }
    }
    __syncthreads();
  }
  if (row < rn) {
#pragma unroll
    for (int u = 0; u < KG_P / 4; ++u) {
      const int j = g + 4 * u;
      if (j < p) Zc[(r0 + row) + (int64_t)j * s] = acc[u];
    }
  }
}

// Omega of every block of a level (s x p row-major, the reference's fill
// order) to the column-major W the product reads.
__global__ void k_h_omega(int64_t s, int p, int nblk, const double* om, double* W) {
  const int64_t tot = (int64_t)nblk * s * p;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % s, j = (e / s) % p;
    W[e] = om[i * p + j];
  }
}

// After the SVD Z = K(C, R) Q = U2 diag(sv) Vt2 (Q^T A = Vt2^T diag(sv)
// U2^T): V (k x s, ld k) = U2(:, :k)^T and S = diag(sv(:k)) of every block
// of a level.
__global__ void k_h_finish_v(int64_t s, int p, int k, int nblk, const double* U2, const double* sv, double* V,
                             double* S) {
  const int64_t totv = (int64_t)nblk * s * k;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < totv; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e / (s * k), rem = e % (s * k);
    const int64_t rr = rem % k, i = rem / k;
    V[e] = U2[c * s * p + i + rr * s];
  }
  const int64_t tots = (int64_t)nblk * k * k;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tots; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e / ((int64_t)k * k), rem = e % ((int64_t)k * k);
    const int rr = (int)(rem % k), cc = (int)(rem / k);
    S[e] = rr == cc ? sv[c * p + rr] : 0.0;
  }
}

// r = b - y (in y), column sums of squares of r and b into nrm[2 c], nrm[2 c + 1]
// (one CTA per column, fixed reduction order).
__global__ void __launch_bounds__(WT) k_h_residual(int64_t n, const double* bb, int64_t ldb, double* y, int64_t ldy,
                                                   double* nrm) {
  __shared__ double red[2][WT / 32];
  const int c = blockIdx.x;
  double sr = 0.0, sb = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += WT) {
    const double bv = bb[i + c * ldb];
    const double rv = bv - y[i + c * ldy];
    y[i + c * ldy] = rv;
    sr += rv * rv;
    sb += bv * bv;
  }
  sr = blr::warp_sum(sr);
  sb = blr::warp_sum(sb);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = sr;
    red[1][threadIdx.x >> 5] = sb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, d = 0.0;
    for (int w = 0; w < WT / 32; ++w) { a += red[0][w]; d += red[1][w]; }
    nrm[2 * c] = a;
    nrm[2 * c + 1] = d;
  }
}

// x += d
__global__ void k_h_axpy(int64_t n, int nrhs, const double* d, int64_t ldd, double* x, int64_t ldx) {
  const int64_t tot = n * nrhs;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % n, c = e / n;
    x[i + c * ldx] += d[i + c * ldd];
  }
}

}  // namespace hk
}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

struct frank_hodlr {
  int64_t n = 0;
  int b = 0, L = 0, k = 0, P = 0;
  int fast = 1;                     // fast_rounded_addition (1) or rounded_addition (0)
  int sm_count = 148;
  cudaStream_t s = nullptr;         // capture stream
  double *D0 = nullptr, *U0 = nullptr, *S0 = nullptr, *V0 = nullptr;
  double *D = nullptr, *U = nullptr, *S = nullptr, *V = nullptr;
  double *Linv = nullptr, *Uinv = nullptr, *UinvT = nullptr;
  int *perm = nullptr, *ipiv = nullptr;
  double* getrf_scratch = nullptr;
  int* geom = nullptr;              // leaf BlrView geometry: off {0, b}, dslot {0}, lslot {-1}
  unsigned long long* flops = nullptr;
  int* err = nullptr;
  int* kfill = nullptr;             // [L + 1][P] ranks, all k (one row per level's stream)
  int* counter = nullptr;           // chunk counters: [2][4 P] of the factorization's two streams, one of the core
  double* Sp = nullptr;             // S' of every internal node's update ([2^L - 1][k x k])
  double* core_part = nullptr;      // [H_NCH][k*k]
  double* Wu = nullptr;             // U_low S' (n/2 x k)
  double* lr_scratch = nullptr;     // addition scratch, one region per level
  int64_t lr_cap = 0;
  std::vector<int64_t> lr_base;     // [L + 1] start of level j's region
  std::vector<cudaStream_t> ls;     // [L + 1] one stream per level for the LowRank additions
  std::vector<cudaEvent_t> lev;     // [L + 1] last addition enqueued on level j's stream
  cudaEvent_t ev_fork = nullptr, ev_core = nullptr;
  double* WZ = nullptr;             // per node: W (lower block's slot) and Z (upper block's slot), U-shaped
  double* Zt = nullptr;             // per node: Zt (upper block's slot), U-shaped
  double* sub[2] = {nullptr, nullptr};   // partial products and T2 of the subtree substitutions (main, side stream)
  cudaStream_t ps = nullptr;        // their substitutions, beside the factorization
  cudaEvent_t ev_pre = nullptr, ev_ps = nullptr;
  ::frank::ops::LrAddTask* tasks_d = nullptr;   // every update's additions, in launch order
  std::vector<::frank::ops::LrAddTask> tasks_h;
  int64_t ntasks_cap = 0;
  double* mv_part = nullptr;
  int64_t mv_part_cap = 0;
  int* mv_counter = nullptr;
  int64_t mv_groups = 0;
  double* work = nullptr;           // refinement: residual / correction (n x nrhs)
  int64_t work_cap = 0;
  double* nrm = nullptr;            // 2 x nrhs
  cudaGraphExec_t gexec = nullptr;
  bool have_A = false, factored = false;
  int64_t launches = 0;
  float factor_ms = 0.f;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
};

namespace {


#define H_TRY(expr)                                                                                         \
  do {                                                                                                      \
    cudaError_t _e = (expr);                                                                                \
    if (_e != cudaSuccess)                                                                                  \
      return ::frank::set_error(FRANK_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e));        \
  } while (0)

int hfail(int code, const std::string& msg) { return ::frank::set_error(code, msg); }

int64_t s_of(const frank_hodlr* h, int l) { return h->n >> l; }
int64_t u_off(const frank_hodlr* h, int l, int c) { return (int64_t)(l - 1) * h->n * h->k + (int64_t)c * s_of(h, l) * h->k; }
int64_t s_off(const frank_hodlr* h, int l, int c) { return ((int64_t)(1 << l) - 2 + c) * h->k * h->k; }
int64_t nblocks_s(const frank_hodlr* h) { return ((int64_t)1 << (h->L + 1)) - 2; }

hk::HView view(const frank_hodlr* h, bool factor) {
  hk::HView v;
  v.n = h->n;
  v.b = h->b;
  v.L = h->L;
  v.k = h->k;
  v.D = factor ? h->D : h->D0;
  v.U = factor ? h->U : h->U0;
  v.S = factor ? h->S : h->S0;
  v.V = factor ? h->V : h->V0;
  return v;
}

hk::LeafFactors leaf_factors(const frank_hodlr* h) {
  return hk::LeafFactors{h->Linv, h->Uinv, h->UinvT, h->perm};
}

// leaf p as a one-block BlrView for the BLR engine's leaf LU and inverse kernels
void leaf_view(const frank_hodlr* h, int p, blr::BlrView<double>& A, blr::FactorWs<double>& ws) {
  A.nb = 1;
  A.bmax = h->b;
  A.kcap = 0;
  A.off = h->geom;
  A.dslot = h->geom + 2;
  A.lslot = h->geom + 3;
  A.rank = nullptr;
  A.D = h->D + (int64_t)p * h->b * h->b;
  A.U = A.S = A.Vt = nullptr;
  std::memset(&ws, 0, sizeof(ws));
  ws.perm = h->perm + (int64_t)p * h->b;
  ws.ipiv = h->ipiv + (int64_t)p * h->b;
  ws.Linv = h->Linv + (int64_t)p * h->b * h->b;
  ws.Uinv = h->Uinv + (int64_t)p * h->b * h->b;
  ws.UinvT = h->UinvT + (int64_t)p * h->b * h->b;
  ws.getrf_scratch = h->getrf_scratch;
  ws.err = h->err;
  ws.flops = h->flops;
}

void enqueue_leaf(frank_hodlr* h, int p, cudaStream_t s) {
  blr::BlrView<double> A;
  blr::FactorWs<double> ws;
  leaf_view(h, p, A, ws);
  const int b = h->b;
  const int np = (b + blr::leaf_width(b) - 1) / blr::leaf_width(b);
  for (int q = 0; q < np; ++q)
    blr::k_leaf_step<double><<<np, blr::leaf_threads(b), blr::leaf_smem(b), s>>>(A, ws, 0, q);
  blr::k_leaf_final<double><<<3 * np, blr::leaf_threads(b), blr::leaf_smem(b), s>>>(A, ws, 0);
  h->launches += np + 1;
}

// LowRank(U_x, S'_node, V_x) (n_node x n_node, U_x ld s(lr), V_x ld k) added
// into node (lr, cr) of the working copy: the dense leaves on stream s, the
// LowRank blocks of each level j on that level's stream (after the node's
// core, event ev_core), so that the additions into blocks needed late (the
// large ones near the top of the node) run beside the factorization of the
// node's first children.
void enqueue_update(frank_hodlr* h, int lr, int cr, const double* Ux, const double* Vx, const double* Sp,
                    cudaStream_t s) {
  const int k = h->k, b = h->b;
  const int64_t sn = s_of(h, lr);
  // Wu = U_x S'
  ::frank::ops::launch_gemm(s, (int)sn, k, k, 1, 1.0, Ux, sn, 0, false, Sp, k, 0, false, 0.0, h->Wu, sn, 0);
  // dense leaves of the node: D_p += Wu(rows of p) V_x(:, cols of p)
  const int nleaf = 1 << (h->L - lr);
  const int pf = cr << (h->L - lr);
  ::frank::ops::launch_gemm(s, b, b, k, nleaf, 1.0, h->Wu, sn, b, false, Vx, k, (int64_t)b * k, false, 1.0,
                            h->D + (int64_t)pf * b * b, b, (int64_t)b * b);
  h->launches += 2;
  // LowRank blocks of the node, one launch per level from the task table
  for (int j = lr + 1; j <= h->L; ++j) {
    const int64_t sj = s_of(h, j);
    const int cbase = cr << (j - lr);
    const int64_t t0 = (int64_t)h->tasks_h.size();
    int64_t off = 0;
    int idx = 0;
    for (int c = cbase; c < cbase + (1 << (j - lr)); ++c, ++idx) {
      ::frank::ops::LrAddTask t;
      t.ua = h->U + u_off(h, j, c);
      t.sa = h->S + s_off(h, j, c);
      t.va = h->V + u_off(h, j, c);
      t.ub = Ux + (int64_t)(c - cbase) * sj;                    // rows of cluster c within the node
      t.sb = Sp;
      t.vb = Vx + (int64_t)((c ^ 1) - cbase) * sj * k;          // columns of its sibling
      t.ldua = sj; t.ldsa = k; t.ldva = k; t.ldub = sn; t.ldsb = k; t.ldvb = k;
      t.scratch_off = h->lr_base[j] + off;
      t.ka = h->kfill + (int64_t)j * h->P + idx;
      t.kb = t.ka;
      t.m = t.n = (int)sj;
      h->tasks_h.push_back(t);
      off += ::frank::ops::lr_add_ws((int)sj, (int)sj, k, k);
    }
    cudaStream_t sj_stream = h->ls[j];
    cudaStreamWaitEvent(sj_stream, h->ev_core, 0);
    ::frank::ops::launch_lr_add_tasks(sj_stream, idx, (int)sj, h->tasks_d + t0, k, h->fast, h->lr_scratch,
                                      h->err + hk::HERR_JACOBI);
    cudaEventRecord(h->lev[j], sj_stream);
    ++h->launches;
  }
}

// Doubles of the partial products and of T2 for `jobs` substitutions of ncols columns.
int64_t sub_part(const frank_hodlr* h, int jobs, int ncols) {
  const int64_t groups = (ncols + hk::HC - 1) / hk::HC;
  int64_t most = 0;
  for (int l = 1; l <= h->L; ++l) most = std::max(most, ((int64_t)1 << l) * hk::h_nch(s_of(h, l)));
  return most * jobs * groups * h->k * hk::HC;
}
int64_t sub_t2(const frank_hodlr* h, int jobs, int ncols) { return (int64_t)h->P * jobs * ncols * h->k; }

// One or two substitutions (hk::HJob) on the subtree (l0, c0), or the H-matvec
// (mode 3, the whole tree): the leaves, then the levels from the bottom up.
// Returns the number of launches.
int enqueue_sub(frank_hodlr* h, const hk::HView& v, int l0, int c0, int njobs, const hk::HJob& j0, const hk::HJob& j1,
                 int ncols, double* buf, int* counter, cudaStream_t s) {
  const int hl = h->L - l0, p0 = c0 << hl, groups = (ncols + hk::HC - 1) / hk::HC;
  double* t2 = buf + sub_part(h, njobs, ncols);
  hk::k_h_leaf_mm<<<dim3(1 << hl, (ncols + hk::HLC - 1) / hk::HLC, njobs), hk::WT, 0, s>>>(v, leaf_factors(h), j0, j1,
                                                                                          p0, ncols);
  for (int l = h->L; l > l0; --l) {
    const int64_t sl = s_of(h, l);
    const int first = c0 << (l - l0);
    const int nodes = j0.mode == 3 ? 1 << l : 1 << (l - l0 - 1);
    hk::k_h_t<<<dim3(hk::h_nch(sl), nodes, njobs * groups), hk::WT, hk::H_TSMEM, s>>>(v, j0, j1, njobs, l, first, ncols,
                                                                                     buf, t2, counter);
    hk::k_h_u<<<dim3((unsigned)((sl + hk::WT - 1) / hk::WT), nodes, njobs * groups), hk::WT, 0, s>>>(
        v, h->WZ, h->Zt, j0, j1, njobs, l, first, ncols, t2);
  }
  return 1 + 2 * (h->L - l0);
}

// A substitution in place on X (col-major), read from src the first time.
hk::HJob sub_job(int mode, const double* src, int64_t srs, int64_t scs, double* X, int64_t ldx) {
  return hk::HJob{mode, src, srs, scs, X, 1, ldx, nullptr, 0};
}

void enqueue_node(frank_hodlr* h, int l, int c, cudaStream_t s) {
  if (l == h->L) {
    enqueue_leaf(h, c, s);
    return;
  }
  const int k = h->k;
  enqueue_node(h, l + 1, 2 * c, s);
  const int up = 2 * c, lo = 2 * c + 1;
  const int64_t sc = s_of(h, l + 1);
  const hk::HView v = view(h, true);
  // the node's own off-diagonal blocks: every addition into them enqueued so
  // far; and the left child's W, Z, Zt
  cudaStreamWaitEvent(s, h->lev[l + 1], 0);
  cudaStreamWaitEvent(s, h->ev_ps, 0);
  // U_up <- L_left^{-1} P U_up (trsm.cpp:106-115 -> 117-125 -> leaves);
  // V_low <- V_low U_left^{-1}, through its transpose in Wu (a leaf writes V_low itself)
  double* Uu = h->U + u_off(h, l + 1, up);
  double* Vl = h->V + u_off(h, l + 1, lo);
  const bool leaf = l + 1 == h->L;
  hk::HJob j0 = sub_job(0, Uu, 1, sc, Uu, sc), j1 = sub_job(1, Vl, k, 1, h->Wu, sc);
  if (leaf) { j1.X = Vl; j1.xrs = k; j1.ldx = 1; }
  h->launches += enqueue_sub(h, v, l + 1, 2 * c, 2, j0, j1, k, h->sub[0], h->counter, s);
  if (!leaf) {
    hk::k_h_transpose<<<dim3((unsigned)((sc + 31) / 32), (k + 31) / 32), hk::WT, 0, s>>>(sc, k, h->Wu, Vl);
    ++h->launches;
  }
  // for the later substitutions, beside the factorization: Z = U_left^{-1} U_up
  cudaEventRecord(h->ev_pre, s);
  cudaStreamWaitEvent(h->ps, h->ev_pre, 0);
  hk::HJob jz = sub_job(2, Uu, 1, sc, h->WZ + u_off(h, l + 1, up), sc);
  h->launches += enqueue_sub(h, v, l + 1, 2 * c, 1, jz, jz, k, h->sub[1], h->counter + 4 * h->P, h->ps);
  // S' = -(S_low V_low)(U_up S_up), one k x k slot per internal node
  double* Sp = h->Sp + ((int64_t)(1 << l) - 1 + c) * k * k;
  hk::k_h_core<<<hk::h_nch(sc), hk::WT, hk::H_TSMEM, s>>>(sc, k, Vl, Uu, h->S + s_off(h, l + 1, lo),
                                                          h->S + s_off(h, l + 1, up), h->core_part, Sp,
                                                          h->counter + 8 * h->P);
  cudaEventRecord(h->ev_core, s);
  ++h->launches;
  enqueue_update(h, l + 1, lo, h->U + u_off(h, l + 1, lo), h->V + u_off(h, l + 1, up), Sp, s);
  enqueue_node(h, l + 1, 2 * c + 1, s);
  // W = M_right(U_low) and Zt = U_right^{-T} V_up^T, once the right child is factored
  cudaEventRecord(h->ev_pre, s);
  cudaStreamWaitEvent(h->ps, h->ev_pre, 0);
  hk::HJob jw = sub_job(0, h->U + u_off(h, l + 1, lo), 1, sc, h->WZ + u_off(h, l + 1, lo), sc);
  hk::HJob jt = sub_job(1, h->V + u_off(h, l + 1, up), k, 1, h->Zt + u_off(h, l + 1, up), sc);
  h->launches += enqueue_sub(h, v, l + 1, 2 * c + 1, 2, jw, jt, k, h->sub[1], h->counter + 4 * h->P, h->ps);
  cudaEventRecord(h->ev_ps, h->ps);
}

int enqueue_factor(frank_hodlr* h, cudaStream_t s) {
  const int64_t nk = (int64_t)h->L * h->n * h->k;
  H_TRY(cudaMemcpyAsync(h->D, h->D0, sizeof(double) * (size_t)h->P * h->b * h->b, cudaMemcpyDeviceToDevice, s));
  H_TRY(cudaMemcpyAsync(h->U, h->U0, sizeof(double) * (size_t)nk, cudaMemcpyDeviceToDevice, s));
  H_TRY(cudaMemcpyAsync(h->V, h->V0, sizeof(double) * (size_t)nk, cudaMemcpyDeviceToDevice, s));
  H_TRY(cudaMemcpyAsync(h->S, h->S0, sizeof(double) * (size_t)nblocks_s(h) * h->k * h->k, cudaMemcpyDeviceToDevice, s));
  H_TRY(cudaMemsetAsync(h->err, 0, sizeof(int) * hk::HERR_SLOTS, s));
  h->launches = 0;
  h->tasks_h.clear();
  H_TRY(cudaEventRecord(h->ev_fork, s));
  H_TRY(cudaStreamWaitEvent(h->ps, h->ev_fork, 0));
  H_TRY(cudaEventRecord(h->ev_ps, h->ps));
  for (int j = 1; j <= h->L; ++j) {
    H_TRY(cudaStreamWaitEvent(h->ls[j], h->ev_fork, 0));
    H_TRY(cudaEventRecord(h->lev[j], h->ls[j]));
  }
  enqueue_node(h, 0, 0, s);
  for (int j = 1; j <= h->L; ++j) {
    H_TRY(cudaEventRecord(h->lev[j], h->ls[j]));
    H_TRY(cudaStreamWaitEvent(s, h->lev[j], 0));
  }
  H_TRY(cudaEventRecord(h->ev_ps, h->ps));
  H_TRY(cudaStreamWaitEvent(s, h->ev_ps, 0));
  H_TRY(cudaGetLastError());
  return FRANK_OK;
}

int check_errors(frank_hodlr* h, cudaStream_t s) {
  int e[hk::HERR_SLOTS];
  H_TRY(cudaMemcpyAsync(e, h->err, sizeof(e), cudaMemcpyDeviceToHost, s));
  H_TRY(cudaStreamSynchronize(s));
  if (e[blr::ERR_SINGULAR_STEP]) return hfail(FRANK_ERR_SINGULAR, "a leaf getrf met a zero pivot");
  if (e[hk::HERR_JACOBI]) return hfail(FRANK_ERR_NOT_CONVERGED, "one-sided Jacobi reached its sweep limit");
  if (e[hk::HERR_RANK]) return hfail(FRANK_ERR_RANK_OVERFLOW, "a recompressed rank exceeded the fixed rank");
  return FRANK_OK;
}

void free_plan(frank_hodlr* h) {
  if (h->gexec) cudaGraphExecDestroy(h->gexec);
  for (void* p : {(void*)h->D0, (void*)h->U0, (void*)h->S0, (void*)h->V0, (void*)h->D, (void*)h->U, (void*)h->S,
                  (void*)h->V, (void*)h->Linv, (void*)h->Uinv, (void*)h->UinvT, (void*)h->perm, (void*)h->ipiv,
                  (void*)h->getrf_scratch, (void*)h->geom, (void*)h->flops, (void*)h->err, (void*)h->kfill,
                  (void*)h->counter, (void*)h->Sp, (void*)h->core_part, (void*)h->Wu, (void*)h->lr_scratch,
                  (void*)h->mv_part, (void*)h->mv_counter, (void*)h->work, (void*)h->nrm, (void*)h->tasks_d})
    if (p) cudaFree(p);
  if (h->e0) cudaEventDestroy(h->e0);
  if (h->e1) cudaEventDestroy(h->e1);
  for (cudaStream_t x : h->ls) if (x) cudaStreamDestroy(x);
  for (cudaEvent_t x : h->lev) if (x) cudaEventDestroy(x);
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  if (h->ev_core) cudaEventDestroy(h->ev_core);
  if (h->ev_pre) cudaEventDestroy(h->ev_pre);
  if (h->ev_ps) cudaEventDestroy(h->ev_ps);
  if (h->ps) cudaStreamDestroy(h->ps);
  for (double* x : {h->WZ, h->Zt, h->sub[0], h->sub[1]}) if (x) cudaFree(x);
  if (h->s) cudaStreamDestroy(h->s);
  delete h;
}

template <typename T>
cudaError_t dalloc(T** p, size_t count) {
  return cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * std::max<size_t>(count, 1));
}

int check_block(const frank_hodlr* h, int l, int c) {
  if (!h) return hfail(FRANK_ERR_INVALID, "null H-matrix");
  if (l < 1 || l > h->L || c < 0 || c >= (1 << l)) return hfail(FRANK_ERR_INVALID, "no such LowRank block");
  return FRANK_OK;
}

// Buffers of the solves and matvecs (nrhs <= HPASS): partial products and T2 of a level, and a
// chunk counter per block and column group (zeroed here, on the stream that the
// launches go to; every launch leaves them zero).
int ensure_mv(frank_hodlr* h, int nrhs, cudaStream_t s) {
  const int64_t need = sub_part(h, 1, nrhs) + sub_t2(h, 1, nrhs);
  const int64_t groups = (nrhs + hk::HC - 1) / hk::HC;
  if (need > h->mv_part_cap) {
    if (h->mv_part) cudaFree(h->mv_part);
    h->mv_part = nullptr;
    h->mv_part_cap = 0;
    H_TRY(dalloc(&h->mv_part, (size_t)need));
    h->mv_part_cap = need;
  }
  if (groups > h->mv_groups) {
    if (h->mv_counter) cudaFree(h->mv_counter);
    h->mv_counter = nullptr;
    h->mv_groups = 0;
    H_TRY(dalloc(&h->mv_counter, (size_t)(groups * h->P)));
    H_TRY(cudaMemsetAsync(h->mv_counter, 0, sizeof(int) * groups * h->P, s));
    h->mv_groups = groups;
  }
  return FRANK_OK;
}

// y = A_H x (FP64), stream-ordered.
int enqueue_matvec(frank_hodlr* h, const double* x, int64_t ldx, double* y, int64_t ldy, int nrhs, cudaStream_t s) {
  int rc = ensure_mv(h, std::min(nrhs, hk::HPASS), s);
  if (rc) return rc;
  for (int c = 0; c < nrhs; c += hk::HPASS) {
    const double* xc = x + c * ldx;
    const hk::HJob j{3, xc, 1, ldx, y + c * ldy, 1, ldy, xc, ldx};
    enqueue_sub(h, view(h, false), 0, 0, 1, j, j, std::min(nrhs - c, hk::HPASS), h->mv_part, h->mv_counter, s);
  }
  H_TRY(cudaGetLastError());
  return FRANK_OK;
}

// passes: 1 = forward (L with the pivots), 2 = backward (U), 3 = both.
int enqueue_solve(frank_hodlr* h, double* d_b, int64_t ldb, int nrhs, cudaStream_t s, int passes = 3) {
  int rc = ensure_mv(h, std::min(nrhs, hk::HPASS), s);
  if (rc) return rc;
  for (int c = 0; c < nrhs; c += hk::HPASS)
    for (int pass = 0; pass < 2; ++pass) {
      if (!(passes & (1 << pass))) continue;
      double* bc = d_b + c * ldb;
      const hk::HJob j = sub_job(pass == 0 ? 0 : 2, bc, 1, ldb, bc, ldb);
      enqueue_sub(h, view(h, true), 0, 0, 1, j, j, std::min(nrhs - c, hk::HPASS), h->mv_part, h->mv_counter, s);
    }
  H_TRY(cudaGetLastError());
  return FRANK_OK;
}

}  // namespace

extern "C" {

int frank_hodlr_create(int64_t n, int leaf, int rank, frank_hodlr** out) {
  if (!out) return hfail(FRANK_ERR_INVALID, "null output pointer");
  *out = nullptr;
  if (leaf < 8 || leaf > hk::HMAX_LEAF || n < 2 * (int64_t)leaf || n % leaf)
    return hfail(FRANK_ERR_INVALID, "H-matrix: need 8 <= leaf <= 512 and n a multiple of leaf, n >= 2 leaf");
  int64_t P = n / leaf;
  int L = 0;
  while (((int64_t)1 << L) < P) ++L;
  if (((int64_t)1 << L) != P || L > 20)
    return hfail(FRANK_ERR_UNSUPPORTED, "H-matrix: n / leaf must be a power of two (binary cluster tree)");
  if (rank < 1 || rank > hk::HMAX_RANK || rank > leaf)
    return hfail(FRANK_ERR_INVALID, "H-matrix: need 1 <= rank <= min(64, leaf)");
  frank_hodlr* h = new frank_hodlr();
  h->n = n;
  h->b = leaf;
  h->L = L;
  h->k = rank;
  h->P = (int)P;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, dev);
  const int64_t nk = (int64_t)L * n * rank, sk = nblocks_s(h) * rank * rank, dd = P * leaf * leaf;
  cudaError_t e = cudaSuccess;
  auto A = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
  A(dalloc(&h->D0, dd)); A(dalloc(&h->D, dd));
  A(dalloc(&h->U0, nk)); A(dalloc(&h->U, nk)); A(dalloc(&h->V0, nk)); A(dalloc(&h->V, nk));
  A(dalloc(&h->S0, sk)); A(dalloc(&h->S, sk));
  A(dalloc(&h->Linv, dd)); A(dalloc(&h->Uinv, dd)); A(dalloc(&h->UinvT, dd));
  A(dalloc(&h->perm, P * leaf)); A(dalloc(&h->ipiv, P * leaf));
  A(dalloc(&h->getrf_scratch, (size_t)blr::leaf_scratch(leaf)));
  A(dalloc(&h->geom, 4)); A(dalloc(&h->flops, blr::FLOP_SLOTS)); A(dalloc(&h->err, hk::HERR_SLOTS));
  A(dalloc(&h->kfill, (size_t)(L + 1) * P)); A(dalloc(&h->counter, 8 * (size_t)P + 1));
  A(dalloc(&h->Sp, (size_t)P * rank * rank)); A(dalloc(&h->core_part, (size_t)hk::H_NCH * rank * rank));
  A(dalloc(&h->Wu, (size_t)(n / 2) * rank));
  // LowRank additions: per level j a scratch region for its largest launch
  // (2^(j-1) blocks of order n >> j, the update of the root's right child),
  // and the task table of all updates
  int64_t cap = 0, ntask = 0;
  h->lr_base.assign(L + 2, 0);
  for (int j = 1; j <= L; ++j) {
    h->lr_base[j] = cap;
    if (j >= 2) cap += ((int64_t)1 << (j - 1)) * ::frank::ops::lr_add_ws((int)(n >> j), (int)(n >> j), rank, rank);
  }
  for (int lr = 1; lr <= L; ++lr) ntask += ((int64_t)1 << (lr - 1)) * (((int64_t)1 << (L - lr + 1)) - 2);
  if (cap > 0) A(dalloc(&h->lr_scratch, (size_t)cap));
  h->lr_cap = cap;
  h->ntasks_cap = ntask;
  A(cudaMalloc(reinterpret_cast<void**>(&h->tasks_d), sizeof(::frank::ops::LrAddTask) * std::max<int64_t>(ntask, 1)));
  h->ls.assign(L + 1, nullptr);
  h->lev.assign(L + 1, nullptr);
  for (int j = 0; j <= L; ++j) {
    A(cudaStreamCreateWithFlags(&h->ls[j], cudaStreamNonBlocking));
    A(cudaEventCreateWithFlags(&h->lev[j], cudaEventDisableTiming));
  }
  A(cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming));
  A(cudaEventCreateWithFlags(&h->ev_core, cudaEventDisableTiming));
  A(cudaEventCreateWithFlags(&h->ev_pre, cudaEventDisableTiming));
  A(cudaEventCreateWithFlags(&h->ev_ps, cudaEventDisableTiming));
  A(cudaStreamCreateWithFlags(&h->ps, cudaStreamNonBlocking));
  A(dalloc(&h->WZ, (size_t)nk)); A(dalloc(&h->Zt, (size_t)nk));
  for (double*& x : h->sub) A(dalloc(&x, (size_t)(sub_part(h, 2, rank) + sub_t2(h, 2, rank))));
  A(cudaStreamCreateWithFlags(&h->s, cudaStreamNonBlocking));
  A(cudaEventCreate(&h->e0));
  A(cudaEventCreate(&h->e1));
  if (e != cudaSuccess) {
    free_plan(h);
    return hfail(FRANK_ERR_CUDA, std::string("H-matrix allocation: ") + cudaGetErrorString(e));
  }
  const int geom[4] = {0, leaf, 0, -1};
  std::vector<int> kf((size_t)(L + 1) * P, rank);
  A(cudaMemcpy(h->geom, geom, sizeof(geom), cudaMemcpyHostToDevice));
  A(cudaMemcpy(h->kfill, kf.data(), sizeof(int) * kf.size(), cudaMemcpyHostToDevice));
  A(cudaMemset(h->counter, 0, sizeof(int) * (8 * (size_t)P + 1)));
  A(cudaMemset(h->flops, 0, sizeof(unsigned long long) * blr::FLOP_SLOTS));
  A(cudaMemset(h->D0, 0, sizeof(double) * dd));
  A(cudaMemset(h->U0, 0, sizeof(double) * nk));
  A(cudaMemset(h->V0, 0, sizeof(double) * nk));
  A(cudaMemset(h->S0, 0, sizeof(double) * sk));
  A(cudaStreamSynchronize(cudaStreamLegacy));   // calls may come on non-blocking streams
  A(cudaFuncSetAttribute(blr::k_leaf_step<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, blr::LEAF_SMEM_MAX));
  A(cudaFuncSetAttribute(blr::k_leaf_final<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, blr::LEAF_SMEM_MAX));
  A(cudaFuncSetAttribute(hk::k_h_t, cudaFuncAttributeMaxDynamicSharedMemorySize, hk::H_TSMEM));
  A(cudaFuncSetAttribute(hk::k_h_core, cudaFuncAttributeMaxDynamicSharedMemorySize, hk::H_TSMEM));
  if (e == cudaSuccess && ::frank::ops::lr_add_prepare() != FRANK_OK) e = cudaErrorInvalidValue;
  if (e != cudaSuccess) {
    free_plan(h);
    return hfail(FRANK_ERR_CUDA, std::string("H-matrix set-up: ") + cudaGetErrorString(e));
  }
  *out = h;
  return FRANK_OK;
}

int frank_hodlr_destroy(frank_hodlr* h) {
  if (h) {
    cudaDeviceSynchronize();
    free_plan(h);
  }
  return FRANK_OK;
}

int frank_hodlr_shape(const frank_hodlr* h, int64_t* n, int* leaf, int* rank, int* levels) {
  if (!h) return hfail(FRANK_ERR_INVALID, "null H-matrix");
  if (n) *n = h->n;
  if (leaf) *leaf = h->b;
  if (rank) *rank = h->k;
  if (levels) *levels = h->L;
  return FRANK_OK;
}

int frank_hodlr_set_lra(frank_hodlr* h, const char* name) {
  if (!h || !name) return hfail(FRANK_ERR_INVALID, "null argument");
  const std::string s(name);
  int fast;
  if (s == "fast_rounded_addition" || s.empty()) fast = 1;
  else if (s == "rounded_addition") fast = 0;
  else return hfail(FRANK_ERR_UNSUPPORTED, "H-matrix: LowRank addition must be fast_rounded_addition or rounded_addition");
  if (fast != h->fast && h->gexec) {
    cudaGraphExecDestroy(h->gexec);
    h->gexec = nullptr;
  }
  h->fast = fast;
  h->factored = false;
  return FRANK_OK;
}

int frank_hodlr_set_dense(frank_hodlr* h, int leaf, const double* a, int64_t ld) {
  if (!h || !a) return hfail(FRANK_ERR_INVALID, "null argument");
  if (leaf < 0 || leaf >= h->P || ld < h->b) return hfail(FRANK_ERR_INVALID, "bad leaf or leading dimension");
  H_TRY(cudaMemcpy2D(h->D0 + (int64_t)leaf * h->b * h->b, sizeof(double) * h->b, a, sizeof(double) * ld,
                     sizeof(double) * h->b, h->b, cudaMemcpyHostToDevice));
  h->have_A = true;
  h->factored = false;
  return FRANK_OK;
}

int frank_hodlr_set_lowrank(frank_hodlr* h, int level, int index, const double* u, const double* s,
                            const double* v) {
  int rc = check_block(h, level, index);
  if (rc) return rc;
  if (!u || !s || !v) return hfail(FRANK_ERR_INVALID, "null argument");
  const int64_t sl = s_of(h, level), k = h->k;
  H_TRY(cudaMemcpy(h->U0 + u_off(h, level, index), u, sizeof(double) * sl * k, cudaMemcpyHostToDevice));
  H_TRY(cudaMemcpy(h->V0 + u_off(h, level, index), v, sizeof(double) * sl * k, cudaMemcpyHostToDevice));
  H_TRY(cudaMemcpy(h->S0 + s_off(h, level, index), s, sizeof(double) * k * k, cudaMemcpyHostToDevice));
  h->have_A = true;
  h->factored = false;
  return FRANK_OK;
}

int frank_hodlr_get_dense(const frank_hodlr* h, int which, int leaf, double* a, int64_t ld) {
  if (!h || !a) return hfail(FRANK_ERR_INVALID, "null argument");
  if (leaf < 0 || leaf >= h->P || ld < h->b) return hfail(FRANK_ERR_INVALID, "bad leaf or leading dimension");
  const double* src = (which ? h->D : h->D0) + (int64_t)leaf * h->b * h->b;
  H_TRY(cudaMemcpy2D(a, sizeof(double) * ld, src, sizeof(double) * h->b, sizeof(double) * h->b, h->b,
                     cudaMemcpyDeviceToHost));
  return FRANK_OK;
}

int frank_hodlr_get_lowrank(const frank_hodlr* h, int which, int level, int index, double* u, double* s, double* v) {
  int rc = check_block(h, level, index);
  if (rc) return rc;
  const int64_t sl = s_of(h, level), k = h->k;
  if (u) H_TRY(cudaMemcpy(u, (which ? h->U : h->U0) + u_off(h, level, index), sizeof(double) * sl * k,
                          cudaMemcpyDeviceToHost));
  if (v) H_TRY(cudaMemcpy(v, (which ? h->V : h->V0) + u_off(h, level, index), sizeof(double) * sl * k,
                          cudaMemcpyDeviceToHost));
  if (s) H_TRY(cudaMemcpy(s, (which ? h->S : h->S0) + s_off(h, level, index), sizeof(double) * k * k,
                          cudaMemcpyDeviceToHost));
  return FRANK_OK;
}

int frank_hodlr_get_pivots(const frank_hodlr* h, int leaf, int* ipiv) {
  if (!h || !ipiv) return hfail(FRANK_ERR_INVALID, "null argument");
  if (leaf < 0 || leaf >= h->P) return hfail(FRANK_ERR_INVALID, "bad leaf");
  if (!h->factored) return hfail(FRANK_ERR_STATE, "getrf has not run");
  H_TRY(cudaMemcpy(ipiv, h->ipiv + (int64_t)leaf * h->b, sizeof(int) * h->b, cudaMemcpyDeviceToHost));
  return FRANK_OK;
}

int frank_hodlr_build_kernel(frank_hodlr* h, int kernel, const double* points, int dim, const double* kparams,
                             void* stream) {
  if (!h || !points) return hfail(FRANK_ERR_INVALID, "null argument");
  if (kernel < 0 || kernel > 3 || dim < 1 || dim > 3) return hfail(FRANK_ERR_INVALID, "bad kernel or dimension");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n = h->n;
  const int k = h->k;
  double* dx = nullptr;
  H_TRY(dalloc(&dx, (size_t)dim * n));
  H_TRY(cudaMemcpy(dx, points, sizeof(double) * dim * n, cudaMemcpyHostToDevice));
  hk::KernelDesc K;
  K.kind = kernel;
  K.dim = dim;
  K.x = dx;
  K.n = n;
  K.p0 = kparams ? kparams[0] : 0.0;
  K.p1 = kparams ? kparams[1] : 0.0;
  hk::k_h_build_leaves<<<4 * h->sm_count, 256, 0, s>>>(K, h->b, h->P, h->D0);
  // LowRank(Dense, rank) on every off-diagonal block, level by level:
  // rsvd (rsvd.cpp:17-29) with sample min(k + 5, s) and the reference's
  // Omega (random_uniform, std::mt19937 seeded 0, functions.cpp:52-66);
  // the block is never stored: Y = A Omega and Z = A^T Q evaluate it tile by tile.
  int rc = FRANK_OK;
  double *W = nullptr, *Y = nullptr, *Q = nullptr, *R = nullptr, *Z = nullptr, *U2 = nullptr, *sv = nullptr,
         *Vt2 = nullptr, *Ur = nullptr, *om = nullptr, *sc = nullptr;
  int* errd = h->err;
  const int64_t pmax = std::min<int64_t>(k + 5, n / 2);   // the widest sample: that of the largest blocks
  const size_t slab = (size_t)n * pmax;   // one level: 2^l blocks of s_l x p
  cudaError_t e = cudaSuccess;
  auto A = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
  int64_t ws_max = 0;
  for (int l = 1; l <= h->L; ++l) {
    const int64_t sl = s_of(h, l);
    const int p = (int)std::min<int64_t>(k + 5, sl);
    ws_max = std::max(ws_max, std::max(::frank::ops::qr_ws((int)sl, p), ::frank::ops::svd_scratch(p, p)) << l);
  }
  A(dalloc(&W, slab)); A(dalloc(&Y, slab)); A(dalloc(&Q, slab)); A(dalloc(&Z, slab)); A(dalloc(&U2, slab));
  A(dalloc(&R, (size_t)pmax * pmax << h->L)); A(dalloc(&Vt2, (size_t)pmax * pmax << h->L));
  A(dalloc(&Ur, (size_t)pmax * pmax << h->L));
  A(dalloc(&sv, (size_t)pmax << h->L)); A(dalloc(&om, (size_t)(n / 2) * pmax)); A(dalloc(&sc, (size_t)ws_max));
  A(cudaMemsetAsync(errd, 0, sizeof(int) * hk::HERR_SLOTS, s));
  for (int l = 1; l <= h->L && e == cudaSuccess; ++l) {
    const int64_t sl = s_of(h, l);
    const int p = (int)std::min<int64_t>(k + 5, sl);
    const int nb = 1 << l;
    std::vector<double> omh((size_t)sl * p);
    {
      std::mt19937 gen;
      gen.seed(0);
      std::uniform_real_distribution<double> dist(0.0, 1.0);
      for (auto& x : omh) x = dist(gen);
    }
    A(cudaMemcpyAsync(om, omh.data(), sizeof(double) * omh.size(), cudaMemcpyHostToDevice, s));
    hk::k_h_omega<<<4 * h->sm_count, 256, 0, s>>>(sl, p, nb, om, W);
    hk::k_h_kgemm<<<dim3((unsigned)((sl + 63) / 64), nb), hk::WT, 0, s>>>(K, sl, p, 0, W, Y);
    ::frank::ops::launch_qr(s, (int)sl, p, nb, Y, sl, sl * p, Q, sl, sl * p, R, p, (int64_t)p * p, sc,
                            ::frank::ops::qr_ws((int)sl, p));
    hk::k_h_kgemm<<<dim3((unsigned)((sl + 63) / 64), nb), hk::WT, 0, s>>>(K, sl, p, 1, Q, Z);
    // Z = A^T Q = Qz Rz, Rz = Ur diag(sv) Vt2: the SVD of the small Rz only
    // (Q^T A = Vt2^T diag(sv) (Qz Ur)^T)
    ::frank::ops::launch_qr(s, (int)sl, p, nb, Z, sl, sl * p, U2, sl, sl * p, R, p, (int64_t)p * p, sc,
                            ::frank::ops::qr_ws((int)sl, p));
    ::frank::ops::launch_svd(s, p, p, nb, R, p, (int64_t)p * p, Ur, p, (int64_t)p * p, sv, p, Vt2, p,
                             (int64_t)p * p, sc, ::frank::ops::svd_scratch(p, p), errd + hk::HERR_JACOBI);
    ::frank::ops::launch_gemm(s, (int)sl, p, p, nb, 1.0, U2, sl, sl * p, false, Ur, p, (int64_t)p * p, false, 0.0, Z,
                              sl, sl * p);
    // U = Q Vt2(:k, :)^T, V = (Qz Ur)(:, :k)^T, S = diag(sv(:k))
    ::frank::ops::launch_gemm(s, (int)sl, k, p, nb, 1.0, Q, sl, sl * p, false, Vt2, p, (int64_t)p * p, true, 0.0,
                              h->U0 + u_off(h, l, 0), sl, sl * k);
    hk::k_h_finish_v<<<4 * h->sm_count, 256, 0, s>>>(sl, p, k, nb, Z, sv, h->V0 + u_off(h, l, 0),
                                                     h->S0 + s_off(h, l, 0));
    A(cudaGetLastError());
    A(cudaStreamSynchronize(s));
  }
  A(cudaStreamSynchronize(s));
  for (void* ptr : {(void*)W, (void*)Y, (void*)Q, (void*)R, (void*)Z, (void*)U2, (void*)sv, (void*)Vt2, (void*)Ur,
                    (void*)om, (void*)sc, (void*)dx})
    if (ptr) cudaFree(ptr);
  if (e != cudaSuccess) return hfail(FRANK_ERR_CUDA, std::string("H-matrix construction: ") + cudaGetErrorString(e));
  int eh[hk::HERR_SLOTS];
  H_TRY(cudaMemcpy(eh, errd, sizeof(eh), cudaMemcpyDeviceToHost));
  if (eh[hk::HERR_JACOBI]) rc = hfail(FRANK_ERR_NOT_CONVERGED, "one-sided Jacobi reached its sweep limit");
  h->have_A = true;
  h->factored = false;
  return rc;
}

int frank_hodlr_getrf(frank_hodlr* h, void* stream) {
  if (!h) return hfail(FRANK_ERR_INVALID, "null H-matrix");
  if (!h->have_A) return hfail(FRANK_ERR_STATE, "H-matrix has no blocks");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!h->gexec) {
    H_TRY(cudaStreamSynchronize(s));
    H_TRY(cudaStreamBeginCapture(h->s, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue_factor(h, h->s);
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(h->s, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (ce != cudaSuccess) return hfail(FRANK_ERR_CUDA, std::string("H-LU capture: ") + cudaGetErrorString(ce));
    const cudaError_t ie = cudaGraphInstantiate(&h->gexec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) return hfail(FRANK_ERR_CUDA, std::string("H-LU graph: ") + cudaGetErrorString(ie));
    if ((int64_t)h->tasks_h.size() > h->ntasks_cap) return hfail(FRANK_ERR_INVALID, "H-LU: task table overflow");
    if (!h->tasks_h.empty())
      H_TRY(cudaMemcpy(h->tasks_d, h->tasks_h.data(), sizeof(::frank::ops::LrAddTask) * h->tasks_h.size(),
                       cudaMemcpyHostToDevice));
  }
  H_TRY(cudaEventRecord(h->e0, s));
  H_TRY(cudaGraphLaunch(h->gexec, s));
  H_TRY(cudaEventRecord(h->e1, s));
  int rc = check_errors(h, s);
  H_TRY(cudaEventElapsedTime(&h->factor_ms, h->e0, h->e1));
  h->factored = rc == FRANK_OK;
  return rc;
}

int frank_hodlr_solve_device(frank_hodlr* h, double* d_b, int64_t ldb, int nrhs, void* stream) {
  if (!h || !d_b) return hfail(FRANK_ERR_INVALID, "null argument");
  if (nrhs < 1 || ldb < h->n) return hfail(FRANK_ERR_INVALID, "bad right-hand sides");
  if (!h->factored) return hfail(FRANK_ERR_STATE, "solve before getrf");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc = enqueue_solve(h, d_b, ldb, nrhs, s);
  if (rc) return rc;
  H_TRY(cudaStreamSynchronize(s));
  return FRANK_OK;
}

int frank_hodlr_trsm_device(frank_hodlr* h, int uplo, double* d_b, int64_t ldb, int nrhs, void* stream) {
  if (!h || !d_b) return hfail(FRANK_ERR_INVALID, "null argument");
  if (nrhs < 1 || ldb < h->n || (uplo != FRANK_LOWER && uplo != FRANK_UPPER))
    return hfail(FRANK_ERR_INVALID, "bad right-hand sides or triangle");
  if (!h->factored) return hfail(FRANK_ERR_STATE, "trsm before getrf");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc = enqueue_solve(h, d_b, ldb, nrhs, s, uplo == FRANK_LOWER ? 1 : 2);
  if (rc) return rc;
  H_TRY(cudaStreamSynchronize(s));
  return FRANK_OK;
}

int frank_hodlr_matvec_device(frank_hodlr* h, const double* d_x, int64_t ldx, double* d_y, int64_t ldy, int nrhs,
                              void* stream) {
  if (!h || !d_x || !d_y) return hfail(FRANK_ERR_INVALID, "null argument");
  if (nrhs < 1 || ldx < h->n || ldy < h->n) return hfail(FRANK_ERR_INVALID, "bad vectors");
  if (!h->have_A) return hfail(FRANK_ERR_STATE, "H-matrix has no blocks");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc = enqueue_matvec(h, d_x, ldx, d_y, ldy, nrhs, s);
  if (rc) return rc;
  H_TRY(cudaStreamSynchronize(s));
  return FRANK_OK;
}

int frank_hodlr_refine_device(frank_hodlr* h, const double* d_b, int64_t ldb, double* d_x, int64_t ldx, int nrhs,
                              double tol, int max_iter, int* iters, double* relres, void* stream) {
  if (!h || !d_b || !d_x) return hfail(FRANK_ERR_INVALID, "null argument");
  if (nrhs < 1 || ldb < h->n || ldx < h->n || max_iter < 0) return hfail(FRANK_ERR_INVALID, "bad arguments");
  if (!h->factored) return hfail(FRANK_ERR_STATE, "refine before getrf");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t need = h->n * nrhs;
  if (need > h->work_cap) {
    if (h->work) cudaFree(h->work);
    if (h->nrm) cudaFree(h->nrm);
    h->work = nullptr;
    h->nrm = nullptr;
    H_TRY(dalloc(&h->work, (size_t)need));
    H_TRY(dalloc(&h->nrm, 2 * (size_t)nrhs));
    h->work_cap = need;
  }
  // x0 = (LU)^{-1} b, then x += (LU)^{-1} (b - A_H x) until every column's
  // relative residual is below tol
  H_TRY(cudaMemcpy2DAsync(d_x, sizeof(double) * ldx, d_b, sizeof(double) * ldb, sizeof(double) * h->n, nrhs,
                          cudaMemcpyDeviceToDevice, s));
  int rc = enqueue_solve(h, d_x, ldx, nrhs, s);
  if (rc) return rc;
  std::vector<double> nr(2 * (size_t)nrhs);
  double worst = 0.0;
  int it = 0;
  for (;; ++it) {
    rc = enqueue_matvec(h, d_x, ldx, h->work, h->n, nrhs, s);
    if (rc) return rc;
    hk::k_h_residual<<<nrhs, hk::WT, 0, s>>>(h->n, d_b, ldb, h->work, h->n, h->nrm);
    H_TRY(cudaMemcpyAsync(nr.data(), h->nrm, sizeof(double) * nr.size(), cudaMemcpyDeviceToHost, s));
    H_TRY(cudaStreamSynchronize(s));
    worst = 0.0;
    for (int c = 0; c < nrhs; ++c) worst = std::max(worst, std::sqrt(nr[2 * c] / std::max(nr[2 * c + 1], 1e-300)));
    if (worst <= tol || it >= max_iter) break;
    rc = enqueue_solve(h, h->work, h->n, nrhs, s);
    if (rc) return rc;
    hk::k_h_axpy<<<2 * h->sm_count, 256, 0, s>>>(h->n, nrhs, h->work, h->n, d_x, ldx);
  }
  H_TRY(cudaGetLastError());
  if (iters) *iters = it;
  if (relres) *relres = worst;
  return worst <= tol ? FRANK_OK : hfail(FRANK_ERR_NOT_CONVERGED, "H-LU refinement did not reach the tolerance");
}

int frank_hodlr_stats(const frank_hodlr* h, int64_t* launches, double* factor_ms) {
  if (!h) return hfail(FRANK_ERR_INVALID, "null H-matrix");
  if (launches) *launches = h->launches;
  if (factor_ms) *factor_ms = h->factor_ms;
  return FRANK_OK;
}

}  // extern "C"
