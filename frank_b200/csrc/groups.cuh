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
constexpr int GQ = 16;   // widest panel
struct GrpShared {
  double G[GQ * GQ];     // V^T V of a panel (strictly upper part)
  double T[GQ * GQ];     // its T factor
  double tau[GQ], beta[GQ], scal[GQ];
  double part[9 * GQ];       // warps' partial sums of a column step, and its row
  double coef[GQ + 2];       // its update coefficients
};

// C (m x n, ldc) = alpha A B + beta C over k, element (i, kk) of A at A[i sai +
// kk sak], (kk, j) of B at B[j sbj + kk sbk].
// Long inner dimension and a small output (bases against bases: k = b, m and n
// ranks): every warp of a slice index q takes an eighth of k for all tiles, so
// each operand row is read once per tile and the warps have equal work; the
// eight partial products go to part (G_PART doubles, in L2) and are summed in
// order.  Otherwise a tile per warp with the whole inner dimension.  Tile shapes
// are the ones with the fewest tensor-pipe cycles and do not change the order in
// which an element is summed.  That order depends on the sizes, and in a slice on
// whether both operands are 16-byte aligned, not on the group's size (from eight
// warps) or on where the operands lie; callers align a matrix the same way wherever
// they put it.
constexpr int G_SLICE_TILES = 81;            // 8 x 8 tiles of a sliced output
constexpr int G_PART = 8 * 64 * G_SLICE_TILES;

// Four consecutive values in FP64 by 16-byte loads.
FRANK_D void load4(const double* p, double (&v)[4]) {
  const double2 x = *reinterpret_cast<const double2*>(p), y = *reinterpret_cast<const double2*>(p + 2);
  v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
FRANK_D void load4(const float* p, double (&v)[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}

// acc = A^T B over rows [k0, k1), both with contiguous rows and 16-byte aligned
// columns: lane t of a quad takes rows 4 t .. 4 t + 3 of every 16 (the products
// of a 16-row block may be summed in any order as long as A and B agree), so a
// load covers 64 bytes of a column instead of 32 (FP32: 16); the L1 looks up
// one line per column and load, and that was what bound these products.
template <int MI, int NI, typename TA, typename TB>
FRANK_D void warp_dgemm_tn(int m, int n, int k0, int k1, const TA* A, int64_t lda, const TB* B, int64_t ldb, int i0,
                           int j0, double (&acc)[MI][NI][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const TA* pa[MI];
  const TB* pb[NI];
#pragma unroll
  for (int i = 0; i < MI; ++i) pa[i] = A + (int64_t)min(i0 + 8 * i + g, m - 1) * lda + k0 + 4 * t;
#pragma unroll
  for (int j = 0; j < NI; ++j) pb[j] = B + (int64_t)min(j0 + 8 * j + g, n - 1) * ldb + k0 + 4 * t;
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  constexpr int U = MI + NI <= 2 ? 4 : (MI + NI <= 4 ? 2 : 1);   // 16-row blocks in flight
  int kk = k0;
  for (; kk + 16 * U <= k1; kk += 16 * U) {
    double a[U][MI][4], b[U][NI][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < MI; ++i) load4(pa[i] + 16 * u, a[u][i]);
#pragma unroll
      for (int j = 0; j < NI; ++j) load4(pb[j] + 16 * u, b[u][j]);
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) pa[i] += 16 * U;
#pragma unroll
    for (int j = 0; j < NI; ++j) pb[j] += 16 * U;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < NI; ++j) dmma884(acc[i][j], a[u][i][v], b[u][j][v]);
  }
  for (; kk < k1; kk += 16) {
    double a[MI][4], b[NI][4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const bool in = kk + 4 * t + v < k1;
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i][v] = in ? double(pa[i][v]) : 0.0;
#pragma unroll
      for (int j = 0; j < NI; ++j) b[j][v] = in ? double(pb[j][v]) : 0.0;
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) pa[i] += 16;
#pragma unroll
    for (int j = 0; j < NI; ++j) pb[j] += 16;
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) dmma884(acc[i][j], a[i][v], b[j][v]);
  }
}

template <typename TA>
FRANK_D bool aligned4(const TA* p, int64_t ld) {
  return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)(ld * (int64_t)sizeof(TA))) & 15) == 0;
}

template <int MI, int NI, typename TA, typename TB>
FRANK_D void g_slices(const Grp& g, int m, int n, int k, const TA* A, int64_t sai, int64_t sak, const TB* B,
                      int64_t sbj, int64_t sbk, int tot, double* part) {
  const int lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
  const int kc = ((k + 7) / 8 + 15) & ~15, q = g.wid & 7, sub = g.wid >> 3, nsub = g.nw >> 3;
  const int k0 = min(k, q * kc), k1 = min(k, k0 + kc);
  const int tm = (m + 8 * MI - 1) / (8 * MI), tn = (n + 8 * NI - 1) / (8 * NI);
  const bool vec = sak == 1 && sbk == 1 && aligned4(A, sai) && aligned4(B, sbj);
  double* pq = part + q * tot;
  for (int tile = sub; tile < tm * tn; tile += nsub) {
    const int i0 = (tile % tm) * 8 * MI, j0 = (tile / tm) * 8 * NI;
    double acc[MI][NI][2];
    if (vec) warp_dgemm_tn<MI, NI>(m, n, k0, k1, A, sai, B, sbj, i0, j0, acc);
    else warp_dgemm_acc<MI, NI, false>(m, n, k0, k1, A, sai, sak, B, sbj, sbk, i0, j0, acc);
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const int r = i0 + 8 * i + gr, c = j0 + 8 * j + 2 * t;
        if (r < m && c < n) pq[r + c * m] = acc[i][j][0];
        if (r < m && c + 1 < n) pq[r + (c + 1) * m] = acc[i][j][1];
      }
  }
}

template <typename TA, typename TB, typename TC>
FRANK_D void g_mm(const Grp& g, int m, int n, int k, double alpha, const TA* A, int64_t sai, int64_t sak, const TB* B,
                  int64_t sbj, int64_t sbk, double beta, TC* C, int64_t ldc, double* part) {
  if (m <= 0 || n <= 0) { g.sync(); return; }
  const int m8 = (m + 7) / 8, n8 = (n + 7) / 8;
  auto cost = [&](int mi, int ni) {
    return ((m8 + mi - 1) / mi) * ((n8 + ni - 1) / ni) * (4 * mi * ni + mi + ni);
  };
  if (m8 * n8 <= G_SLICE_TILES && k >= 128 && g.nw >= 8) {
    const int c33 = cost(3, 3), c22 = cost(2, 2), c11 = cost(1, 1);
    const int tot = m * n;
    if (c33 <= c22 && c33 <= c11) g_slices<3, 3>(g, m, n, k, A, sai, sak, B, sbj, sbk, tot, part);
    else if (c22 <= c11) g_slices<2, 2>(g, m, n, k, A, sai, sak, B, sbj, sbk, tot, part);
    else g_slices<1, 1>(g, m, n, k, A, sai, sak, B, sbj, sbk, tot, part);
    g.sync();
    for (int e = g.tid; e < tot; e += g.nt) {
      double v[8], s = 0.0;
#pragma unroll
      for (int x = 0; x < 8; ++x) v[x] = part[e + x * tot];
#pragma unroll
      for (int x = 0; x < 8; ++x) s += v[x];
      dgemm_store(C + e % m + (int64_t)(e / m) * ldc, s, alpha, beta);
    }
    g.sync();
    return;
  }
  auto rounds = [&](int mi, int ni) {
    const int tiles = ((m8 + mi - 1) / mi) * ((n8 + ni - 1) / ni);
    return ((tiles + g.nw - 1) / g.nw) * (4 * mi * ni + mi + ni);
  };
  const int c42 = rounds(4, 2), c23 = rounds(2, 3), c11 = rounds(1, 1);
  if (c42 <= c23 && c42 <= c11)
    warps_dgemm<4, 2>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  else if (c23 <= c11)
    warps_dgemm<2, 3>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  else
    warps_dgemm<1, 1>(g.wid, g.nw, m, n, k, alpha, A, sai, sak, B, sbj, sbk, beta, C, ldc);
  g.sync();
}

// Householder reflector (dlarfg) of a column with leading entry alpha and
// squared norm n2 = alpha^2 + (squared norm below it): v = [1; x scal],
// H = I - tau v v^T, H x = beta e_1.  One reciprocal square root and one
// reciprocal (every warp forms them, so the FP64 pipe pays for each): with
// h = |alpha| + ||x||, tau = h / ||x|| and scal = sign / h.
// FINE: a Newton step each on the norm and its reciprocal, to half a unit in the last
// place, on which H's orthogonality rests.  The additions of single blocks, whose
// results are the factors themselves, take it (2 to 5 % closer to 64 bits); a
// factorization does not show it and would take 3 % longer (n = 8192 at 1e-8).
template <bool FINE>
FRANK_D void reflector(double alpha, double n2, double& beta, double& tau, double& scal) {
  double rn = rsqrt(n2), nrm = n2 * rn;
  const double aa = fabs(alpha);
  if (FINE) {
    nrm = fma(0.5 * rn, fma(-nrm, nrm, n2), nrm);
    rn = fma(rn, fma(-nrm, rn, 1.0), rn);
  }
  const double rh = __drcp_rn(aa + nrm);
  beta = alpha >= 0.0 ? -nrm : nrm;
  tau = fma(aa, rn, 1.0);
  scal = alpha >= 0.0 ? rh : -rh;
}

// Householder QR (dgeqr2 conventions) of a panel P (m x n, ldp, n <= W, n <= m),
// rows in registers: thread t of the first eight warps holds rows t, t + 256,
// ... (RPT of them, m <= 256 RPT) of all W columns.  A column step is one
// reduction of the column's dot products with every column -- later ones for
// the update, itself for the norm, earlier ones for the T factor -- which a
// warp does by recursive halving (W sums in W + 1 exchanges instead of 5 W);
// the warps' sums meet in shared memory, where one warp forms the reflector.  Kept in shared memory instead, a
// 512 x 16 panel of both sides was bound by its bandwidth (256 KB a step:
// 51 us; 3.3 us a column).  On return V (clean, unit lower trapezoid, ldv)
// holds the reflectors (V may be P), s.T the T factor (upper, zero below) and
// R (n x n, ldr) the triangle with zeros below its diagonal.
template <int W, int RPT, bool FINE>
static __device__ __noinline__ void panel_qr_rows(Grp g, int m, int n, const double* P, int64_t ldp, double* V, int64_t ldv, double* R,
                           int64_t ldr, GrpShared& s) {
  const int lane = threadIdx.x & 31;
  const bool on = g.wid < 8;
  double a[RPT][W];
#pragma unroll
  for (int k = 0; k < RPT; ++k)
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const int r = g.tid + 256 * k;
      a[k][c] = (on && r < m && c < n) ? P[r + c * ldp] : 0.0;
    }
  for (int j = 0; j < n; ++j) {
    double* part = s.part;                         // [8][GQ] warp sums, [GQ] row j
    double x[RPT], f[W];
    if (on) {
      // column j of the rows below j (by selection: registers have no index)
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        double v = a[k][0];
#pragma unroll
        for (int c = 1; c < W; ++c) v = j == c ? a[k][c] : v;
        x[k] = g.tid + 256 * k > j ? v : 0.0;
      }
      double d[W];
#pragma unroll
      for (int c = 0; c < W; ++c) {
        d[c] = x[0] * a[0][c];
#pragma unroll
        for (int k = 1; k < RPT; ++k) d[c] = fma(x[k], a[k][c], d[c]);
      }
      if (g.tid == j) {
#pragma unroll
        for (int c = 0; c < W; ++c) part[8 * GQ + c] = a[0][c];
      }
      // recursive halving: lane l ends with the sum of column l % W
#pragma unroll
      for (int h = W / 2; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int c = 0; c < h; ++c) {
          const double send = up ? d[c] : d[c + h], keep = up ? d[c + h] : d[c];
          d[c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
      }
#pragma unroll
      for (int h = W; h < 32; h <<= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], h);
      if (lane < W) part[g.wid * GQ + lane] = d[0];
    }
    g.sync();
    // one warp turns the sums into the reflector and the step's coefficients
    // (eight of them doing it would cost the FP64 pipe more than a barrier)
    if (g.wid == 0) {
      const int c = lane & (W - 1);
      double q[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) q[w] = part[w * GQ + c];
      const double top = part[8 * GQ + c];
      const double dot = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
      const double alpha = __shfl_sync(0xffffffffu, top, j), xn2 = __shfl_sync(0xffffffffu, dot, j);
      double beta = alpha, tau = 0.0, scal = 0.0;
      if (xn2 > 0.0) reflector<FINE>(alpha, fma(alpha, alpha, xn2), beta, tau, scal);
      const double w = fma(scal, dot, top);
      if (lane < j) s.G[lane + j * GQ] = s.scal[lane] * w;
      else if (lane == j) { s.tau[j] = tau; s.beta[j] = beta; s.scal[j] = scal; }
      if (lane < W) s.coef[lane] = c > j && c < n ? tau * w : 0.0;
      if (lane == 0) s.coef[GQ] = scal;
    }
    g.sync();
    if (!on) continue;
    // rows above j of R are final; row j: a_jc - tau w
    const double scal = s.coef[GQ];
#pragma unroll
    for (int cc = 0; cc < W; ++cc) f[cc] = s.coef[cc];
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const double xs = g.tid + 256 * k == j ? 1.0 : x[k] * scal;
#pragma unroll
      for (int cc = 0; cc < W; ++cc) a[k][cc] = fma(-f[cc], xs, a[k][cc]);
    }
  }
  g.sync();
  // T = (triu(G, 1) + diag(1 / tau))^{-1}: lane = row, a column per warp and
  // pass, back substitution with the solved value by shuffle (tau_s multiplies
  // where the inverse would divide; tau = 0 gives a zero row and column)
  {
    const double tr = lane < n ? s.tau[lane] : 0.0;
    for (int c = g.wid; c < n; c += g.nw) {
      double up = lane == c ? 1.0 : 0.0;
      for (int q = c; q >= 0; --q) {
        const double xq = __shfl_sync(0xffffffffu, up * tr, q);
        if (lane < q) up = fma(-s.G[lane + q * GQ], xq, up);
        else if (lane == q) up = xq;
      }
      if (lane < GQ) s.T[lane + c * GQ] = lane <= c ? up : 0.0;
    }
  }
  if (on) {
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int r = g.tid + 256 * k;
#pragma unroll
      for (int c = 0; c < W; ++c)
        if (r < m && c < n) {
          if (r < n) R[r + c * ldr] = r < c ? a[k][c] : (r == c ? s.beta[c] : 0.0);
          V[r + c * ldv] = r > c ? a[k][c] * s.scal[c] : (r == c ? 1.0 : 0.0);
        }
    }
  }
  g.sync();
}

// Widest panel of m rows: 16 columns of up to two rows a thread, 8 of up to four.
FRANK_HD int panel_width(int m) { return m <= 512 ? 16 : 8; }

template <bool FINE = false>
FRANK_D void g_panel_qr(const Grp& g, int m, int n, const double* P, int64_t ldp, double* V, int64_t ldv, double* R,
                        int64_t ldr, GrpShared& s) {
  if (m > 512) panel_qr_rows<8, 4, FINE>(g, m, n, P, ldp, V, ldv, R, ldr, s);
  else if (m > 256) panel_qr_rows<16, 2, FINE>(g, m, n, P, ldp, V, ldv, R, ldr, s);
  else panel_qr_rows<16, 1, FINE>(g, m, n, P, ldp, V, ldv, R, ldr, s);
}

FRANK_HD int panel_ld(int m) { return ((m + 15) & ~15) + 4; }   // 4 mod 16: conflict-free fragments

// Scratch of the blocked routines: W, W2 (GQ x widest operand each) and the
// partial products, in global memory.
struct GrpScratch {
  double *W, *W2, *part;
};

// Trailing products of a panel V (mr x jn, ldv, clean) with its T: X (mr x r,
// ldx) -= V op(T) V^T X; rows of X at or below kr are zero on entry.
FRANK_D void g_wy(const Grp& g, int mr, int kr, int jn, const double* V, int64_t ldv, const double* T, bool tt, int r,
                  double* X, int64_t ldx, const GrpScratch& x) {
  for (int op = 0; op < 3; ++op) {
    // W = V^T X; W2 = op(T) W; X -= V W2
    const double* A = op == 1 ? T : V;
    const int64_t ld = op == 1 ? GQ : ldv;
    const bool ta = op == 0 || (op == 1 && tt);
    const double* B = op == 0 ? X : (op == 1 ? x.W : x.W2);
    double* C = op == 0 ? x.W : (op == 1 ? x.W2 : X);
    g_mm(g, op == 2 ? mr : jn, r, op == 0 ? kr : jn, op == 2 ? -1.0 : 1.0, A, ta ? ld : 1, ta ? 1 : ld, B,
         op == 0 ? ldx : GQ, 1, op == 2 ? 1.0 : 0.0, C, op == 2 ? ldx : GQ, x.part);
  }
}

// Blocked Householder QR of A (m x n, lda; overwritten): panels of w <= panel_width(m)
// columns, T factors in Tf (GQ x GQ per panel), the clean V of panel p in rows
// and columns j0 .. of V (ldv; may be A), R (min(m, n) x n, ldr, zeros below the
// diagonal) apart.  The trailing products read the panel from smP (shared,
// panel_ld(m) x w doubles), or from A where that is in shared memory (smP null).
FRANK_D void g_qr(const Grp& g, int m, int n, double* A, int64_t lda, double* V, int64_t ldv, double* R, int64_t ldr,
                  double* Tf, int w, double* smP, GrpShared& s, const GrpScratch& x) {
  const int km = min(m, n), lane = threadIdx.x & 31;
  for (int j0 = 0, p = 0; j0 < km; j0 += w, ++p) {
    const int jn = min(w, km - j0), mr = m - j0, nc = n - j0 - jn;
    double* Ap = A + j0 + (int64_t)j0 * lda;
    double* At = Ap + (int64_t)jn * lda;
    double* Vp = smP ? smP : Ap;
    const int64_t ldp = smP ? panel_ld(m) : lda;
    // R below this panel's diagonal block is zero
    for (int c = g.wid; c < jn; c += g.nw)
      for (int r = j0 + jn + lane; r < km; r += 32) R[r + (int64_t)(j0 + c) * ldr] = 0.0;
    g_panel_qr(g, mr, jn, Ap, lda, Vp, ldp, R + j0 + (int64_t)j0 * ldr, ldr, s);
    for (int c = g.wid; c < jn; c += g.nw)
#pragma unroll 4
      for (int r = lane; r < mr; r += 32) V[(j0 + r) + (int64_t)(j0 + c) * ldv] = Vp[r + c * ldp];
    for (int e = g.tid; e < GQ * GQ; e += g.nt) Tf[p * GQ * GQ + e] = s.T[e];
    if (nc > 0) {
      g_wy(g, mr, mr, jn, Vp, ldp, s.T, true, nc, At, lda, x);
      // the finished rows of R
      for (int e = g.tid; e < jn * nc; e += g.nt)
        R[(j0 + e % jn) + (int64_t)(j0 + jn + e / jn) * ldr] = At[e % jn + (int64_t)(e / jn) * lda];
    }
    g.sync();
  }
}

// X (m x r, ldx) := Q X with the k reflectors of g_qr (clean V in A, Tf, panels
// of w).  Rows of X at or below nz are zero on entry.
FRANK_D void g_apply_q(const Grp& g, int m, int k, const double* A, int64_t lda, const double* Tf, int w, int r,
                       double* X, int64_t ldx, int nz, const GrpScratch& x) {
  for (int p = (k + w - 1) / w - 1; p >= 0; --p) {
    const int j0 = p * w, kr = min(m - j0, max(0, nz - j0));
    nz = m;
    if (kr == 0) continue;
    g_wy(g, m - j0, kr, min(w, k - j0), A + j0 + (int64_t)j0 * lda, lda, Tf + p * GQ * GQ, false, r, X + j0, ldx, x);
  }
}

// The same QR for any number of rows: a panel goes down the rows in chunks, the
// first of GT_ROWS rows, each later one factored stacked under the panel's
// triangle (flat-tree TSQR; Demmel, Grigori, Hoemmen, Langou,
// "Communication-optimal parallel and sequential QR and LU factorizations",
// SIAM J. Sci. Comput. 34, 2012).  The reflectors of a later chunk are [I; X]
// over the panel's top rows and the chunk, so only X is stored, in the chunk's
// place in A; T factors of panel p, chunk i at Tf + (p * gt_chunks(m) + i)
// GQ^2.  smP: panel_ld(min(m, GT_ROWS)) x GQ doubles (shared).
constexpr int GT_ROWS = 512;
FRANK_HD int gt_chunks(int m) { return m <= GT_ROWS ? 1 : 1 + (m - GT_ROWS + GT_ROWS - GQ - 1) / (GT_ROWS - GQ); }

// X (rows [0, jn) at Xt, chunk rows at Xc, ldx) <- (I - [I; V] op(T) [I; V]^T) X
FRANK_D void g_wy_stacked(const Grp& g, int mr, int kr, int jn, const double* V, int64_t ldv, const double* T, bool tt,
                          int r, double* Xt, double* Xc, int64_t ldx, const GrpScratch& x) {
  for (int e = g.tid; e < jn * r; e += g.nt) x.W[e % jn + (e / jn) * GQ] = Xt[e % jn + (int64_t)(e / jn) * ldx];
  g.sync();
  for (int op = 0; op < 3; ++op) {
    const double* A = op == 1 ? T : V;
    const int64_t ld = op == 1 ? GQ : ldv;
    const bool ta = op == 0 || (op == 1 && tt);
    const double* B = op == 0 ? Xc : (op == 1 ? x.W : x.W2);
    double* C = op == 0 ? x.W : (op == 1 ? x.W2 : Xc);
    if (op == 0 && kr <= 0) continue;
    g_mm(g, op == 2 ? mr : jn, r, op == 0 ? kr : jn, op == 2 ? -1.0 : 1.0, A, ta ? ld : 1, ta ? 1 : ld, B,
         op == 0 ? ldx : GQ, 1, op == 1 ? 0.0 : 1.0, C, op == 2 ? ldx : GQ, x.part);
  }
  for (int e = g.tid; e < jn * r; e += g.nt) Xt[e % jn + (int64_t)(e / jn) * ldx] -= x.W2[e % jn + (e / jn) * GQ];
  g.sync();
}

FRANK_D void g_qr_tall(const Grp& g, int m, int n, double* A, int64_t lda, double* R, int64_t ldr, double* Tf,
                       double* smP, GrpShared& s, const GrpScratch& x) {
  const int km = min(m, n), lane = threadIdx.x & 31, nch = gt_chunks(m), ldp = panel_ld(min(m, (int)GT_ROWS));
  for (int j0 = 0, p = 0; j0 < km; j0 += GQ, ++p) {
    const int jn = min((int)GQ, km - j0), nc = n - j0 - jn;
    for (int c = g.wid; c < jn; c += g.nw)
      for (int r = j0 + jn + lane; r < km; r += 32) R[r + (int64_t)(j0 + c) * ldr] = 0.0;
    double* Rp = R + j0 + (int64_t)j0 * ldr;
    double* Ct = A + j0 + (int64_t)(j0 + jn) * lda;      // the panel's rows of the later columns
    int row = j0;
    for (int i = 0; row < m; ++i) {
      const int cr = min(m - row, i == 0 ? (int)GT_ROWS : GT_ROWS - GQ);
      double* Ac = A + row + (int64_t)j0 * lda;
      const int top = i == 0 ? 0 : jn;                   // stacked rows of the triangle
      if (i > 0) {
        for (int c = g.wid; c < jn; c += g.nw) {
          if (lane < jn) smP[lane + c * ldp] = lane <= c ? Rp[lane + (int64_t)c * ldr] : 0.0;
#pragma unroll 4
          for (int r = lane; r < cr; r += 32) smP[jn + r + c * ldp] = Ac[r + (int64_t)c * lda];
        }
        g.sync();
        g_panel_qr<true>(g, jn + cr, jn, smP, ldp, smP, ldp, Rp, ldr, s);
      } else {
        g_panel_qr<true>(g, cr, jn, Ac, lda, smP, ldp, Rp, ldr, s);
      }
      double* T = Tf + (int64_t)(p * nch + i) * GQ * GQ;
      for (int c = g.wid; c < jn; c += g.nw)
#pragma unroll 4
        for (int r = lane; r < cr; r += 32) Ac[r + (int64_t)c * lda] = smP[top + r + c * ldp];
      for (int e = g.tid; e < GQ * GQ; e += g.nt) T[e] = s.T[e];
      if (nc > 0) {
        if (i == 0) g_wy(g, cr, cr, jn, smP, ldp, s.T, true, nc, Ct, lda, x);
        else g_wy_stacked(g, cr, cr, jn, smP + jn, ldp, s.T, true, nc, Ct, Ac + (int64_t)jn * lda, lda, x);
      }
      g.sync();
      row += cr;
    }
    for (int e = g.tid; e < jn * nc; e += g.nt)
      R[(j0 + e % jn) + (int64_t)(j0 + jn + e / jn) * ldr] = Ct[e % jn + (int64_t)(e / jn) * lda];
    g.sync();
  }
}

// X (m x r, ldx) := Q X with the k reflectors of g_qr_tall; rows of X at or below
// nz are zero on entry.
FRANK_D void g_apply_q_tall(const Grp& g, int m, int k, const double* A, int64_t lda, const double* Tf, int r,
                            double* X, int64_t ldx, int nz, const GrpScratch& x) {
  const int nch = gt_chunks(m);
  for (int p = (k + GQ - 1) / GQ - 1; p >= 0; --p) {
    const int j0 = p * GQ, jn = min((int)GQ, k - j0);
    const int c0 = min(m - j0, (int)GT_ROWS);
    const int later = m - j0 - c0, nl = (later + GT_ROWS - GQ - 1) / (GT_ROWS - GQ);
    for (int i = nl; i >= 1; --i) {
      const int row = j0 + c0 + (i - 1) * (GT_ROWS - GQ), cr = min(m - row, GT_ROWS - GQ);
      g_wy_stacked(g, cr, min(cr, nz - row), jn, A + row + (int64_t)j0 * lda, lda,
                   Tf + (int64_t)(p * nch + i) * GQ * GQ, false, r, X + j0, X + row, ldx, x);
    }
    // top rows: chunk 0 holds them all the same (they may be filled by the later chunks)
    g_wy(g, c0, min(c0, max(nz - j0, jn)), jn, A + j0 + (int64_t)j0 * lda, lda, Tf + (int64_t)p * nch * GQ * GQ, false,
         r, X + j0, ldx, x);
    nz = m;
  }
}

// Project the columns of Y (m x p, ldy) out of the span of Q (m x k, element (i,
// j) at Q[i qi + j qj], orthonormal columns), twice (classical Gram-Schmidt
// with one re-orthogonalisation): Z (k x p, ldz) = Q^T Y_0, Y = (I - Q Q^T)^2 Y_0,
// Y_0 = Q Z + Y.  Z2 (k x p) is scratch.
template <typename T>
FRANK_D void g_project_out(const Grp& g, int m, int k, int p, const T* Q, int64_t qi, int64_t qj, double* Y,
                           int64_t ldy, double* Z, int64_t ldz, double* Z2, const GrpScratch& x) {
  for (int op = 0; op < 4; ++op) {
    const bool tn = !(op & 1);
    double* Zp = op >= 2 ? Z2 : Z;
    const int64_t ldp = op >= 2 ? k : ldz;
    g_mm(g, tn ? k : m, p, tn ? m : k, tn ? 1.0 : -1.0, Q, tn ? qj : qi, tn ? qi : qj, tn ? Y : Zp, tn ? ldy : ldp, 1,
         tn ? 0.0 : 1.0, tn ? Zp : Y, tn ? ldp : ldy, x.part);
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
template <bool FINE = false>
FRANK_D int g_rrqr(const Grp& g, int m, int n, double* A, int lda, double thr, int maxr, double* tau,
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
    // the pivot's remaining norm is the search's own maximum
    const double* x = A + kp * lda;
    const double alpha = x[r];
    double bt = 0.0, t = 0.0, sc = 0.0;
    if (mx > 0.0) reflector<FINE>(alpha, mx, bt, t, sc);
    bv = -1.0;
    bi = -1;
    for (int c0 = 0; c0 < n; c0 += ng) {
      const int c = c0 + gi;
      const bool live = c < n && c != kp && at[min(c, n - 1)] > r;
      double* p = A + min(c, n - 1) * lda;
      double d0 = 0.0;
#pragma unroll 4
      for (int e = r + 1 + l8; e < m; e += 8) d0 = fma(x[e], p[e], d0);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) d0 += __shfl_xor_sync(0xffffffffu, d0, o);
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

constexpr int G_COLS_MAX = 160;   // rows the register columns of g_apply_cols hold
FRANK_D void g_apply_rrqr(const Grp& g, int m, int k, int r, const double* A, int lda, const double* tau,
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

FRANK_D int g_rand_qrcp(const Grp& g, int m, int n, double* A, int64_t lda, double* R, int64_t ldr,
                                        double thr, int maxr, int w, int* jpvt, double* Tf, double* om, double* nrm2,
                                        double* region, int* iscr, unsigned long long* mx, GrpShared& s,
                                        const GrpScratch& x) {
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
    g_mm(g, sb, nr, mr, 1.0, om, 1, sb, At, lda, 1, 0.0, Y, ldy, x.part);
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
        for (int e = r + b + lane; e < min(m, n); e += 32) R[e + (int64_t)(r + c) * ldr] = 0.0;
      g_panel_qr(g, mr, b, At, lda, smP, ldp, Rp, ldr, s);
      for (int c = g.wid; c < b; c += g.nw)
#pragma unroll 4
        for (int e = lane; e < mr; e += 32) At[e + (int64_t)c * lda] = smP[e + c * ldp];
      for (int e = g.tid; e < GQ * GQ; e += g.nt) Tf[(int64_t)panel * GQ * GQ + e] = s.T[e];
      const int nc = nr - b;
      if (nc > 0) {
        double* Ac = At + (int64_t)b * lda;
        g_wy(g, mr, mr, b, smP, ldp, s.T, true, nc, Ac, lda, x);
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
        // |h| <= tol ||g_p|| ||g_q||: nothing to rotate (squared while the squares are in range)
        const double ab = a * b;
        if (!on || a == 0.0 || b == 0.0) continue;
        if (ab > 1e-280 && ab < 1e280 ? h * h <= tol * tol * ab : fabs(h) <= tol * sqrt(a) * sqrt(b)) continue;
        const double zeta = (b - a) / (2.0 * h);
        const double za = fabs(zeta), zc = fmin(za, 1e100), u = fma(zc, zc, 1.0);
        const double t = copysign(__drcp_rn(za + u * rsqrt(u)), zeta);
        const double f = fma(t, t, 1.0);
        double c = rsqrt(f);
        c = fma(0.5 * c, fma(-f * c, c, 1.0), c);
        const double s = c * t;
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
