// dense.cu -- FP64 dense block operations of the batched solver:
//   k_gram        [G | H] = W^H [W | Y]  (partials over row chunks)
//   k_gram_reduce fixed-order sum of the partials, Hermitian completion
//   (small.cu: from G and H to the Ritz values, the rotation's coefficients C
//   and the next Chebyshev window)
//   k_rotate      V = W C
//   k_residual64_cols  R = (-Delta) V - V diag(theta) (FP64 stencil), S = -2 c_hop R
//                 (FP32), residual partial sums (k_residual64, one thread per site
//                 and column, with LAPH_RESID_KERNEL=0)
//   k_resid       residual norms, convergence mask
// Columns [0, c0) of a problem (whole tiles of locked Ritz vectors) are frozen:
// the Gram skips frozen x frozen tiles, the small problem projects the active
// block against them, and the rotation and residual write active columns only.
// These replace SLEPc's BV orthogonalisation and DS dense eigensolve inside
// EPSSolve (src/ev_ts.cpp:263).  tcgen05 has no FP64 kind, so the Gram and the
// rotation run on the FP64 tensor path of mma.sync (four real MMAs per complex
// product): at the same peak as the FP64 FMA pipe, but one instruction per 256
// FMAs (m8n8k4, the rotation) or 2048 (m16n8k16, the Gram), which measured
// 7-10% faster for each kernel than FMA, and the Gram another 9% on m16n8k16.
#include "batch.cuh"
#include "dense.cuh"
#include "filter.cuh"
#include "stencil64cols.cuh"

namespace laph {

// d(8x8, 2 per thread) += a(8x4, 1 per thread) b(4x8, 1 per thread), FP64 tensor MMA.
// Not volatile: a pure function of its operands, so the compiler may schedule
// it; the callers issue the MMAs of one k-step accumulator-major (all tiles'
// first product, then all tiles' second, ...) so that consecutive MMAs never
// feed the same accumulator and the tensor pipe does not wait on its latency.
__device__ __forceinline__ void dmma884(double (&acc)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(acc[0]), "+d"(acc[1])
      : "d"(a), "d"(b));
}
// d(16x8, 4 per thread) += a(16x16, 8 per thread) b(16x8, 4 per thread), FP64 tensor MMA: the same peak as
// m8n8k4 (37.1 TFLOP/s measured for both on this part) with an eighth of the instructions.  Fragments, g =
// lane / 4, t = lane % 4: a[r] = A(g + 8 (r & 1), t + 4 (r >> 1)); b[r] = B(t + 4 r, g); d[0..1] = D(g, 2t + {0,1}),
// d[2..3] = D(g + 8, 2t + {0,1}).
__device__ __forceinline__ void dmma16816(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}

// ------------------------------------------------------------------ Gram ---
// CTA: 64 threads, output tiles G[ti,tj] = W_ti^H W_tj and H[ti,tj] = W_ti^H Y_tj
// (32 x 32 each, as 2 x 4 m16n8k16 tiles; warp 0 forms G, warp 1 H), over the rows of one chunk; the
// W_ti tile is staged once for both products.  Rows arrive through a
// two-stage cp.async ring (dynamic shared memory [stage][A|W|Y][col][GP], row q of column c at
// c GP + (q ^ 4 (c & 1)): the 16-byte fragment reads of a quarter warp, two columns of one parity pair,
// then fall on eight different bank groups),
// so the next 16 rows load while the current 16 are multiplied.
constexpr int GT = 32, GK = 16, GP = GK;
__device__ __forceinline__ int gsw(int c, int q) { return c * GP + (q ^ ((c & 1) << 2)); }
constexpr int kGramSmem = 2 * 3 * GT * GP * (int)sizeof(double2);

__global__ void __launch_bounds__(64) k_gram(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                             const int* __restrict__ start, int np, int chunk_rows,
                                             const double2* __restrict__ W, const double2* __restrict__ Y,
                                             double2* __restrict__ gpart) {
  const int p = find_prob(start, np, blockIdx.x);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int T = d.k / GT;
  const int npair = T * (T + 1) / 2;
  int t = blockIdx.x - start[p];
  const int chunk = t / npair;
  const int pair = t - chunk * npair;
  int pr = pair, ti = 0;
  while (pr >= T - ti) {
    pr -= T - ti;
    ++ti;
  }
  const int tj = LAPH_IX(ti + pr, T);
  if ((tj + 1) * GT <= ps[p].c0) return;  // both tiles frozen: not needed
  const double2* A = W + d.blk + (size_t)(ti * GT) * d.dim;
  const double2* BW = W + d.blk + (size_t)(tj * GT) * d.dim;
  const double2* BY = Y + d.blk + (size_t)(tj * GT) * d.dim;
  const int r0 = chunk * chunk_rows, r1 = min(d.dim, r0 + chunk_rows);
  extern __shared__ double2 gsm[];
  // thread -> (column c, row q) of each staged 32 x 16 slab: 16 threads per column, 256 B contiguous
  auto load = [&](int r, int b) {
    double2* s = gsm + b * 3 * GT * GP;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int idx = threadIdx.x + 64 * e;
      const int c = idx >> 4, q = idx & 15;
      const int row = r + q;
      const bool ok = row < r1;
      const size_t off = (size_t)c * d.dim + (ok ? row : 0);
      cp_async16(s + LAPH_IX(gsw(c, q), GT * GP), A + off, ok);
      cp_async16(s + gsw(GT + c, q), BW + off, ok);
      cp_async16(s + gsw(2 * GT + c, q), BY + off, ok);
    }
    cp_async_commit();
  };
  // FP64 tensor path: warp 0 forms G = W_ti^H W_tj, warp 1 H = W_ti^H Y_tj, each
  // as 2 x 4 tiles of m16n8k16 (one MMA per tile and stage of 16 rows);
  // conj(w) b = (wr br + wi bi) + i (wr bi - wi br), the last as wi (-br)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  double accr[2][4][4], acci[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) accr[i][j][e] = acci[i][j][e] = 0.0;
  const int nstep = (r1 - r0 + GK - 1) / GK;
  // On a diagonal tile pair (ti == tj) the reduction keeps only the upper
  // triangle (G and H are Hermitian): the 16x8 tiles entirely below the
  // diagonal (rows 16-31 x columns 0-15) are skipped, 2 of 8 per warp.
  const bool diag = ti == tj;
  load(r0, 0);
  for (int it = 0; it < nstep; ++it) {
    const int b = it & 1;
    if (it + 1 < nstep) {
      load(r0 + (it + 1) * GK, b ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double2* sA = gsm + b * 3 * GT * GP;
    const double2* sB = sA + (1 + warp) * GT * GP;  // W_tj or Y_tj
    // A fragments (m16 x k16, row = column of W_ti, k = row of the stage): a[r] at (g + 8 (r & 1), t4 + 4 (r >> 1))
    double ar[2][8], ai[2][8];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double2 a = sA[gsw(16 * i + g + 8 * (r & 1), t4 + 4 * (r >> 1))];
        ar[i][r] = a.x;
        ai[i][r] = a.y;
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // B fragment (k16 x n8): b[r] at (t4 + 4 r, g)
      double br[4], bi[4], bn[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const double2 v = sB[gsw(8 * j + g, t4 + 4 * r)];
        br[r] = v.x;
        bi[r] = v.y;
        bn[r] = -v.x;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (!diag || !(i == 1 && j < 2)) dmma16816(accr[i][j], ar[i], br);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (!diag || !(i == 1 && j < 2)) dmma16816(acci[i][j], ar[i], bi);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (!diag || !(i == 1 && j < 2)) dmma16816(accr[i][j], ai[i], bi);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (!diag || !(i == 1 && j < 2)) dmma16816(acci[i][j], ai[i], bn);
    }
    __syncthreads();
  }
  // partial layout: [chunk][which][pair][32*32]; C fragment rows g (+8), columns 2 t4 + {0, 1}
  double2* o = gpart + d.gp + ((size_t)(chunk * 2 + warp) * npair + pair) * (GT * GT);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int rb = 2 * i + h;  // 8-row block of the output
        if (diag && rb > j) continue;
#pragma unroll
        for (int e = 0; e < 2; ++e)
          o[(16 * i + 8 * h + g) * GT + 8 * j + 2 * t4 + e] = make_double2(accr[i][j][2 * h + e], acci[i][j][2 * h + e]);
      }
}


// The same partial products for batches with few (tile pair, chunk) units: there
// the two warps of a unit run 16 MMA tiles' chains on two of an SM's four FP64
// tensor pipes, 2 us per 16-row stage however idle the chip is (647 us for the
// 250 stages of 11^3).  Here a CTA of four warps takes a 32 x 16 half of G or of H
// of a unit, one m16n8k16 tile per warp: four times the CTAs, a quarter of the
// chain on each pipe, and a six-stage ring so that the loads run ahead of the
// shorter stages.  Every output element sees the same MMAs in the same order.
constexpr int GSS = 6, kGramSplitStage = (GT + GT / 2) * GP;  // stages; double2 per stage
// Up to this many units (of 32^3: 6 timeslices of block width 160, 3 of 224).  Four Rayleigh-Ritz steps, ms, merged ->
// split: 11^3 k 64 (3 units) 3.41 -> 1.86, 16^3 k 96 (12) 6.17 -> 2.98, 24^3 k 160 (90) 9.74 -> 7.29, 24^3 x 6 (540)
// 19.6 -> 18.7; a mixed batch of 990 units 85 -> 80 ms per solve; 2160 units (32^3 x 12) and 2952 (48^3 x 2, k 256):
// no difference or 1% the other way, for twice the reads from L2.
constexpr int kGramSplitUnits = 1200;
constexpr int kGramSplitSmem = GSS * kGramSplitStage * (int)sizeof(double2);

__global__ void __launch_bounds__(128) k_gram_split(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                                    const int* __restrict__ start, int np, int chunk_rows,
                                                    const double2* __restrict__ W, const double2* __restrict__ Y,
                                                    double2* __restrict__ gpart) {
  const int unit = blockIdx.x >> 2, which = (blockIdx.x >> 1) & 1, half = blockIdx.x & 1;
  const int p = find_prob(start, np, unit);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int T = d.k / GT;
  const int npair = T * (T + 1) / 2;
  const int t = unit - start[p];
  const int chunk = t / npair;
  const int pair = t - chunk * npair;
  int pr = pair, ti = 0;
  while (pr >= T - ti) {
    pr -= T - ti;
    ++ti;
  }
  const int tj = LAPH_IX(ti + pr, T);
  if ((tj + 1) * GT <= ps[p].c0) return;  // both tiles frozen: not needed
  const double2* A = W + d.blk + (size_t)(ti * GT) * d.dim;
  const double2* B = (which ? Y : W) + d.blk + (size_t)(tj * GT + half * (GT / 2)) * d.dim;
  const int r0 = chunk * chunk_rows, r1 = min(d.dim, r0 + chunk_rows);
  extern __shared__ double2 gsm[];
  auto load = [&](int st) {
    double2* s = gsm + (st % GSS) * kGramSplitStage;
    const int row = r0 + st * GK + (threadIdx.x & 15);
    const bool ok = row < r1;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const int c = (threadIdx.x >> 4) + 8 * e;  // 32 columns of W_ti, then 16 of W_tj or Y_tj
      const double2* src = e < 4 ? A + (size_t)c * d.dim : B + (size_t)(c - GT) * d.dim;
      cp_async16(s + LAPH_IX(gsw(c, threadIdx.x & 15), kGramSplitStage), src + (ok ? row : 0), ok);
    }
    cp_async_commit();
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int i = warp & 1, j = warp >> 1;  // 16-row and 8-column tile of this warp
  const bool skip = ti == tj && i == 1 && half == 0;  // entirely below the diagonal: not kept
  double accr[4] = {0.0, 0.0, 0.0, 0.0}, acci[4] = {0.0, 0.0, 0.0, 0.0};
  const int nstep = (r1 - r0 + GK - 1) / GK;
#pragma unroll
  for (int st = 0; st < GSS - 1; ++st) {
    if (st < nstep) load(st);
    else cp_async_commit();
  }
  for (int it = 0; it < nstep; ++it) {
    cp_async_wait<GSS - 2>();
    __syncthreads();
    if (it + GSS - 1 < nstep) load(it + GSS - 1);
    else cp_async_commit();
    if (skip) continue;
    const double2* sA = gsm + (it % GSS) * kGramSplitStage;
    double ar[8], ai[8], br[4], bi[4], bn[4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const double2 a = sA[gsw(16 * i + g + 8 * (r & 1), t4 + 4 * (r >> 1))];
      ar[r] = a.x;
      ai[r] = a.y;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const double2 v = sA[gsw(GT + 8 * j + g, t4 + 4 * r)];
      br[r] = v.x;
      bi[r] = v.y;
      bn[r] = -v.x;
    }
    dmma16816(accr, ar, br);
    dmma16816(acci, ar, bi);
    dmma16816(accr, ai, bi);
    dmma16816(acci, ai, bn);
  }
  cp_async_wait<0>();
  if (skip) return;
  double2* o = gpart + d.gp + ((size_t)(chunk * 2 + which) * npair + pair) * (GT * GT);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (ti == tj && 2 * i + h > 2 * half + j) continue;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      o[(16 * i + 8 * h + g) * GT + 16 * half + 8 * j + 2 * t4 + e] = make_double2(accr[2 * h + e], acci[2 * h + e]);
  }
}

// Sum partials (fixed order) and complete the Hermitian matrices G, H
// (column-major k x k at kk and kk + k*k).
__global__ void k_gram_reduce(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                              const int* __restrict__ start, int np, const double2* __restrict__ gpart,
                              double2* __restrict__ GH) {
  const int p = find_prob(start, np, blockIdx.x);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int T = d.k / GT, npair = T * (T + 1) / 2;
  const int e = (blockIdx.x - start[p]) * blockDim.x + threadIdx.x;
  if (e >= 2 * npair * GT * GT) return;
  const int tile = e / (GT * GT), w = e - tile * GT * GT;
  const int which = tile / npair;
  int pr = tile - which * npair, ti = 0;
  while (pr >= T - ti) {
    pr -= T - ti;
    ++ti;
  }
  const int tj = ti + pr;
  if ((tj + 1) * GT <= ps[p].c0) return;  // frozen tile pair: not computed
  double2 s = make_double2(0.0, 0.0);
  for (int c = 0; c < d.nchunk; ++c) s = cadd(s, gpart[d.gp + ((size_t)(c * 2 + which) * npair + tile - which * npair) * (GT * GT) + w]);
  const int i = ti * GT + w / GT, j = tj * GT + w % GT;
  double2* M = GH + d.kk + (size_t)which * d.k * d.k;
  if (ti == tj) {
    // diagonal tile holds both triangles; keep the upper one and mirror it
    if (i <= j) {
      if (i == j) s.y = 0.0;
      M[i + (size_t)j * d.k] = s;
      M[j + (size_t)i * d.k] = cconj(s);
    }
  } else {
    M[i + (size_t)j * d.k] = s;
    M[j + (size_t)i * d.k] = cconj(s);
  }
}

// ------------------------------------------------- Chebyshev coefficients --
// Scaled recurrence for a filter of degree m (chosen by the host each
// iteration).  With E_1 = S/2, E_0 = 0 and
//   E_{n+1} = 2B E_n - E_{n-1} + T_n(theta_B) S,
// T_m(B) V = V T_m(Theta_B) + E_m exactly (S = 2(BV - V Theta_B)).  Each
// column is carried as E'_n = E_n / nu_n, nu_n = max(1, |T_n|), so every FP32
// value stays O(|S|):
//   step 1: E'_2 = (B S + T_1 S) / nu_2
//   step 2: E'_3 = (2 nu_2 B E'_2 + (T_2 - 1/2) S) / nu_3
//   step n: E'_{n+1} = (2 nu_n B E'_n - nu_{n-1} E'_{n-1} + T_n S) / nu_{n+1}
//   final : W' = (T_m / nu_m) V + E'_m   (= W / nu_m)
// A direct pass (ProbState::direct) filters V itself: S holds V in FP32
// (k_direct_start) and X_n = T_n(B) V, carried as X'_n = X_n / nu_n:
//   step 1: X'_1 = B S / nu_1
//   step 2: X'_2 = (2 nu_1 B X'_1 - S) / nu_2
//   step n: X'_n = (2 nu_{n-1} B X'_{n-1} - nu_{n-2} X'_{n-2}) / nu_n   (no S)
//   final : W' = X'_{m-1}   (T_m / nu_m = 0: the pass applies T_{m-1}(B))
__global__ void k_coef(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps, int np,
                       const double* __restrict__ theta, double* __restrict__ tcoef, double* __restrict__ scol, int m,
                       const int* __restrict__ dm) {
  if (dm) m = *dm;  // degree decided on the device (the device-side loop)
  const int p = blockIdx.x;
  if (p >= np || !ps[p].active) return;
  const ProbDesc d = pd[p];
  const ProbState S = ps[p];
  const int k = d.k;
  const double* th = theta + d.kv;
  double* tc = tcoef + d.tc;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const double tb = 1.0 + 2.0 * (S.lam_cut - th[j]) / (S.lam_max - S.lam_cut);
    double tn[kMaxFilterDeg + 2], nu[kMaxFilterDeg + 2];
    tn[0] = 1.0;
    tn[1] = tb;
    for (int n = 2; n <= m; ++n) tn[n] = 2.0 * tb * tn[n - 1] - tn[n - 2];
    for (int n = 0; n <= m; ++n) nu[n] = fmax(1.0, fabs(tn[n]));
    if (S.direct) {
      for (int n = 1; n < m; ++n) {
        const double a = n == 1 ? 1.0 / nu[1] : 2.0 * nu[n - 1] / nu[n];
        const double z = n >= 3 ? -nu[n - 2] / nu[n] : 0.0;
        const double g = n == 2 ? -1.0 / nu[2] : 0.0;
        tc[((size_t)n * 3 + 0) * k + j] = a;
        tc[((size_t)n * 3 + 1) * k + j] = z;
        tc[((size_t)n * 3 + 2) * k + j] = g;
      }
      tc[((size_t)m * 3 + 0) * k + j] = 0.0;
      scol[d.kv + j] = -2.0 * S.c_hop;
      continue;
    }
    for (int n = 1; n < m; ++n) {
      double a, z, g;
      if (n == 1) {
        a = 1.0 / nu[2];
        z = 0.0;
        g = tn[1] / nu[2];
      } else if (n == 2) {
        a = 2.0 * nu[2] / nu[3];
        z = 0.0;
        g = (tn[2] - 0.5) / nu[3];
      } else {
        a = 2.0 * nu[n] / nu[n + 1];
        z = -nu[n - 1] / nu[n + 1];
        g = tn[n] / nu[n + 1];
      }
      tc[((size_t)n * 3 + 0) * k + j] = a;
      tc[((size_t)n * 3 + 1) * k + j] = z;
      tc[((size_t)n * 3 + 2) * k + j] = g;
    }
    tc[((size_t)m * 3 + 0) * k + j] = tn[m] / nu[m];
    scol[d.kv + j] = -2.0 * S.c_hop;
  }
}

// ---------------------------------------------------------------- rotate ---
constexpr int RR = 128, RC = 32, RK = 8, RS = 3;
constexpr int kRotStage = RK * RR + RK * RC;  // double2 per stage
constexpr int kRotSmem = RS * kRotStage * (int)sizeof(double2);

// V = W C on the FP64 tensor path (mma.sync m8n8k4 f64): CTA tile 128 rows x
// 32 columns, W and C slabs of RK columns/rows through a three-stage cp.async
// ring (dynamic shared memory), each warp a 32 x 32 sub-tile of 4 x 4 8x8 MMA
// tiles; the complex product as four real MMAs (Vr += Wr Cr - Wi Ci,
// Vi += Wr Ci + Wi Cr).  Against the same tile on the FP64 FMA pipe (8 x 4
// complex per thread, 246 registers): +7% for the dense phase.
__global__ void __launch_bounds__(128) k_rotate(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                                     const int* __restrict__ start, int np,
                                                     const double2* __restrict__ Wp, const double2* __restrict__ KK,
                                                     double2* __restrict__ Vp) {
  const int p = find_prob(start, np, blockIdx.x);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int nct = d.k / RC;
  const int t = blockIdx.x - start[p];
  const int rt = t / nct, ct = t - rt * nct;
  const int row0 = rt * RR, col0 = ct * RC;
  if (col0 < ps[p].c0) return;  // frozen columns keep their Ritz vectors
  const int k = d.k;
  const double2* C = KK + d.kk + 4 * (size_t)k * k;  // the small step's output
  const double2* Wb = Wp + d.blk;
  extern __shared__ double2 rsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr0 = warp * 32;             // warp's rows within the CTA tile
  const int fr = lane >> 2, fk = lane & 3;  // fragment row / k index
  double accr[4][4][2], acci[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) accr[i][j][0] = accr[i][j][1] = acci[i][j][0] = acci[i][j][1] = 0.0;
  auto load = [&](int q0, int b) {
    double2* sW = rsm + b * kRotStage;
    double2* sC = sW + RK * RR;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int idx = threadIdx.x + 128 * e;
      const int c = idx >> 7, r = idx & 127;
      const int row = row0 + r;
      const bool ok = row < d.dim;
      cp_async16(sW + c * RR + r, Wb + (size_t)LAPH_IX(q0 + c, k) * d.dim + (ok ? row : 0), ok);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int idx = threadIdx.x + 128 * e;
      const int c = idx & 31, r = idx >> 5;
      cp_async16(sC + r * RC + c, C + (size_t)LAPH_IX(col0 + c, k) * k + LAPH_IX(q0 + r, k), true);
    }
    cp_async_commit();
  };
  const int nstep = k / RK;
#pragma unroll
  for (int s = 0; s < RS - 1; ++s) {
    if (s < nstep) load(s * RK, s);
    else cp_async_commit();
  }
  for (int it = 0; it < nstep; ++it) {
    cp_async_wait<RS - 2>();
    __syncthreads();
    if (it + RS - 1 < nstep) load((it + RS - 1) * RK, (it + RS - 1) % RS);
    else cp_async_commit();
    const double2* sW = rsm + (it % RS) * kRotStage;
    const double2* sC = sW + RK * RR;
#pragma unroll
    for (int ks = 0; ks < RK / 4; ++ks) {
      const int q = ks * 4 + fk;
      double ar[4], ai[4], br[4], bi[4], bn[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 a = sW[q * RR + wr0 + 8 * i + fr];  // A(row fr, k fk) of row tile i
        ar[i] = a.x;
        ai[i] = a.y;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 b = sC[q * RC + 8 * j + fr];  // B(k fk, col fr) of column tile j
        br[j] = b.x;
        bi[j] = b.y;
        bn[j] = -b.y;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma884(accr[i][j], ar[i], br[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma884(acci[i][j], ar[i], bi[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma884(accr[i][j], ai[i], bn[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma884(acci[i][j], ai[i], br[j]);
    }
  }
  cp_async_wait<0>();
  // D(row fr, cols 2 fk, 2 fk + 1) of each 8x8 tile
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + wr0 + 8 * i + fr;
    if (row >= d.dim) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = col0 + 8 * j + 2 * fk + e;
        Vp[(size_t)d.blk + (size_t)col * d.dim + row] = make_double2(accr[i][j][e], acci[i][j][e]);
      }
  }
}

// R = A V - V Theta in FP64 (A = -Delta), S = -2 c_hop R in FP32 for the next
// filter, and per-CTA partial sums of |R_j|^2.  One thread per (site,
// column); CTA = 128 sites of one column.
__global__ void __launch_bounds__(128) k_residual64(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                                    const int* __restrict__ start, int np,
                                                    const double2* __restrict__ U64, const double2* __restrict__ Vp,
                                                    const double* __restrict__ theta, float2* __restrict__ Sp,
                                                    double* __restrict__ rpart) {
  const int p = find_prob(start, np, blockIdx.x);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int nst = (d.V3 + 127) >> 7;
  const int t = blockIdx.x - start[p];
  const int st = t % nst, j = t / nst;
  if (j < ps[p].c0) return;  // frozen column: its residual partials stand
  const int s = st * 128 + threadIdx.x;
  double rr = 0.0;
  if (s < d.V3) {
    const Lat g{d.L, d.L * d.L, d.V3};
    const double2* U = U64 + d.u64;
    const size_t col = (size_t)d.blk + (size_t)j * d.dim;
    const double2* x = Vp + col;
    int sx, sy, sz;
    site_xyz(g, s, sx, sy, sz);
    double2 acc[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      const int u = nb_up(g, sx, sy, sz, mu), dn = nb_dn(g, sx, sy, sz, mu);
      double2 xu[3], xd[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        xu[b] = __ldg(x + (size_t)b * d.V3 + u);
        xd[b] = __ldg(x + (size_t)b * d.V3 + dn);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          cfma(acc[a], __ldg(U + (size_t)(mu * 9 + 3 * a + b) * d.V3 + s), xu[b]);
          cfmac(acc[a], __ldg(U + (size_t)(mu * 9 + 3 * b + a) * d.V3 + dn), xd[b]);
        }
    }
    const double th = __ldg(theta + d.kv + j);
    const double sc = -2.0 * ps[p].c_hop;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double2 xs = __ldg(x + (size_t)a * d.V3 + s);
      const double2 r = make_double2((6.0 - th) * xs.x - acc[a].x, (6.0 - th) * xs.y - acc[a].y);
      rr += r.x * r.x + r.y * r.y;
      Sp[col + (size_t)a * d.V3 + s] = make_float2((float)(sc * r.x), (float)(sc * r.y));  // colour-major
    }
  }
  // block reduction (fixed order)
  for (int o = 16; o > 0; o >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, o);
  __shared__ double red[4];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = rr;
  __syncthreads();
  if (threadIdx.x == 0) rpart[d.rp + (size_t)st * d.k + j] = red[0] + red[1] + red[2] + red[3];
}

// The same residual laid out like the FP64 block stencil A W
// (stencil64cols.cuh): CTA = 128 sites x a block of cols columns, NC per thread
// and trip.  Each thread leaves |r|^2 of its site and columns in shared memory
// (FP32: one site's share of a norm needs no more), and one warp sums the 128
// sites of the trip's columns in a fixed order (FP64) into the same per-tile
// partials as the kernel above while the others load the next trip.
constexpr int kResidSmem = kStencil64Smem + kTrip64 * kSites64 * (int)sizeof(float);

template <int NC>
__global__ void __launch_bounds__(kThreads64, 2)
    k_residual64_cols(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps, const int* __restrict__ start,
                      int np, int cols, const double2* __restrict__ U64, const double2* __restrict__ Vp,
                      const double* __restrict__ theta, float2* __restrict__ Sp, double* __restrict__ rpart) {
  const int p = find_prob(start, np, blockIdx.x);
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const int nst = (d.V3 + kSites64 - 1) / kSites64;
  const int t = blockIdx.x - start[p];
  const int st = t % nst, cb = t / nst;
  const int c0 = ps[p].c0;
  const int j0 = cb * cols, j1 = min(d.k, j0 + cols);
  if (j1 <= c0) return;  // frozen columns: their residual partials stand
  const int jstart = max(j0, c0);
  const int i = threadIdx.x % kSites64, grp = threadIdx.x / kSites64;
  // threads past the last site compute the last site again and write nothing
  const bool valid = st * kSites64 + i < d.V3;
  const int s = min(st * kSites64 + i, d.V3 - 1);
  extern __shared__ double2 s64[];
  double2 (*sU)[kSites64] = reinterpret_cast<double2 (*)[kSites64]>(s64);
  float (*sPart)[kSites64] = reinterpret_cast<float (*)[kSites64]>(s64 + 54 * kSites64);
  const Lat g{d.L, d.L * d.L, d.V3};
  int up[3], dn[3], sx, sy, sz;
  site_xyz(g, s, sx, sy, sz);
#pragma unroll
  for (int mu = 0; mu < 3; ++mu) {
    up[mu] = nb_up(g, sx, sy, sz, mu);
    dn[mu] = nb_dn(g, sx, sy, sz, mu);
  }
  load_links64(U64 + d.u64, g, s, dn, sU, i, grp);
  __syncthreads();
  const double sc = -2.0 * ps[p].c_hop;
#pragma unroll 1
  for (int jb = jstart; jb < j1; jb += kGroups64 * NC) {
    const int j = jb + grp * NC;
    float part[NC];
    if (j < j1) {  // uniform over the group
      const size_t col = (size_t)d.blk + (size_t)j * d.dim;
      const double2* x = Vp + col;
      int co[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) co[c] = min(c, j1 - 1 - j) * (int)d.dim;
      double2 acc[NC][3];
      if (i == 0)  // the group's next columns into L2
        for (int c = kGroups64 * NC; c < min((kGroups64 + 1) * NC, j1 - j); ++c)
          prefetch64(x + (size_t)c * d.dim, d.V3, st * kSites64);
      hop64_cols<NC>(sU, i, d.V3, up, dn, x, co, acc);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double th = __ldg(theta + d.kv + LAPH_IX(min(j + c, j1 - 1), d.k));
        double r2 = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double2 xs = __ldg(x + co[c] + a * d.V3 + s);
          const double2 r = make_double2((6.0 - th) * xs.x - acc[c][a].x, (6.0 - th) * xs.y - acc[c][a].y);
          r2 += r.x * r.x + r.y * r.y;
          if (valid && j + c < j1) Sp[col + co[c] + a * d.V3 + s] = make_float2((float)(sc * r.x), (float)(sc * r.y));
        }
        part[c] = valid ? (float)r2 : 0.f;
      }
    }
    __syncthreads();  // the sums of the trip before are done
    if (j < j1)
#pragma unroll
      for (int c = 0; c < NC; ++c) sPart[grp * NC + c][i] = part[c];
    __syncthreads();
    // column c = tid / 4 summed by 4 threads over 32 sites each, then across them
    if (threadIdx.x < 32) {
      const int c = threadIdx.x >> 2, q = threadIdx.x & 3;
      const bool live = c < kGroups64 * NC && jb + c < j1;
      double sum = 0.0;
      if (live)
#pragma unroll 8
        for (int e = 0; e < kSites64 / 4; ++e) sum += (double)sPart[c][q * (kSites64 / 4) + e];
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (q == 0 && live) rpart[d.rp + (size_t)st * d.k + jb + c] = sum;
    }
  }
}

// ------------------------------------------------------- residuals/conv ----
__global__ void k_resid(const ProbDesc* __restrict__ pd, ProbState* __restrict__ ps, const double* __restrict__ rpart,
                        double* __restrict__ resid, double tol, int* __restrict__ n_active) {
  const int p = blockIdx.x;
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  __shared__ double s_max[32];
  __shared__ int s_cnt[32];
  double mx = 0.0;
  int cnt = 0;
  const double lmax = ps[p].lam_max;
  for (int j = threadIdx.x; j < d.k; j += blockDim.x) {
    double s = 0.0;
    for (int r = 0; r < d.nrt; ++r) s += rpart[d.rp + (size_t)r * d.k + j];
    const double rr = sqrt(s) / lmax;
    resid[d.kv + j] = rr;
    if (j < d.nev) {
      mx = fmax(mx, rr);
      cnt += rr <= tol;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_max[threadIdx.x >> 5] = mx;
    s_cnt[threadIdx.x >> 5] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    int c = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      m = fmax(m, s_max[w]);
      c += s_cnt[w];
    }
    ProbState& S = ps[p];
    S.max_resid = m;
    S.nconv = c;
    S.iters += 1;
    // lock the leading columns whose residual is well below tol: the filter
    // leaves them as they are (W_j = V_j); they stay in every Rayleigh-Ritz
    // and are re-measured, so one that drifts up is unlocked next iteration
    int nl = 0;
    while (nl < d.nev && resid[d.kv + nl] <= 0.3 * tol) ++nl;
    S.nlock = nl;
    // frozen block for the Rayleigh-Ritz: whole Gram tiles of locked columns,
    // never shrinking (a frozen column is not re-measured, so it stays locked)
    S.c0 = max(S.c0, min(nl / GT * GT, d.k - GT));
    if (c >= d.nev) S.active = 0;
    else atomicAdd(n_active, 1);
  }
}

// ---------------------------------------------------------------- output ---
// fix_phase (modules/eigensystem.cpp:4-30) on V[:, :nev]: phase_j = arg V(0,j),
// V_j <- e^{-i phase_j} V_j; also |V_j|^2 for tr(V^dag V).  One CTA per column.
__global__ void k_phase_fix(const ProbDesc* __restrict__ pd, const int* __restrict__ start, int np,
                            double2* __restrict__ Vp, double* __restrict__ phases, double* __restrict__ norms,
                            int apply) {
  const int p = find_prob(start, np, blockIdx.x);
  const ProbDesc d = pd[p];
  const int j = blockIdx.x - start[p];
  if (j >= d.nev) return;
  double2* v = Vp + d.blk + (size_t)j * d.dim;
  const double2 v0 = v[0];
  const double ph = atan2(v0.y, v0.x);
  double sn, cs;
  sincos(ph, &sn, &cs);
  const double2 f = apply ? make_double2(cs, -sn) : make_double2(1.0, 0.0);
  double nrm = 0.0;
  __syncthreads();
  for (int i = threadIdx.x; i < d.dim; i += blockDim.x) {
    const double2 x = v[i];
    nrm += x.x * x.x + x.y * x.y;
    if (apply) v[i] = cmul(f, x);
  }
  __shared__ double red[256];
  red[threadIdx.x] = nrm;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    phases[d.kv + j] = ph;
    norms[d.kv + j] = red[0];
  }
}

// ---------------------------------------------------------- start window --
// State of a random start block used without a first Rayleigh-Ritz (window
// from the learned model or fixed): every column gets the Ritz value lam_max,
// where T_n(theta_B) = (-1)^n, so the first filter pass runs entirely through
// the FP32 correction E = T_m(B) V - V T_m(theta_B) (accurate to FP32, which
// is all a first pass needs); the window is the one already in the state.
__global__ void k_start_window(const ProbDesc* __restrict__ pd, ProbState* __restrict__ ps, int np,
                               double* __restrict__ theta) {
  const int p = blockIdx.x;
  if (p >= np) return;
  const ProbDesc d = pd[p];
  ProbState& S = ps[p];
  for (int j = threadIdx.x; j < d.k; j += blockDim.x) theta[d.kv + j] = S.lam_max;
  if (threadIdx.x == 0) {
    double cut = S.lam_cut;
    if (cut >= S.lam_max - 1e-3) cut = S.lam_max - 1e-3;
    if (cut < 1e-6) cut = 1e-6;
    S.lam_cut = cut;
    S.c_hop = 2.0 / (S.lam_max - cut);
    S.c_diag = (S.lam_max + cut - 12.0) / (S.lam_max - cut);
    S.chol_fail = 0;
    S.theta_min = S.lam_max;
  }
}

// --------------------------------------------------------------- output ---
// Colour-major columns (c*V3 + site) -> the reference's 3*site + colour order.
__global__ void k_to_reference(const double2* __restrict__ in, double2* __restrict__ out, int V3, int nev) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V3) return;
  const size_t col = (size_t)blockIdx.y * 3 * V3;
#pragma unroll
  for (int c = 0; c < 3; ++c) out[col + 3 * (size_t)s + c] = __ldg(in + col + (size_t)c * V3 + s);
}

// ------------------------------------------------------------- launchers ---
int start_window(const ProbDesc* pd, ProbState* ps, int np, double* theta, cudaStream_t st) {
  k_start_window<<<np, 256, 0, st>>>(pd, ps, np, theta);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int to_reference(const double2* in, double2* out, int V3, int nev, cudaStream_t st) {
  k_to_reference<<<dim3((V3 + 255) / 256, nev), 256, 0, st>>>(in, out, V3, nev);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int dense_init() {
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_gram_split, cudaFuncAttributeMaxDynamicSharedMemorySize, kGramSplitSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_rotate, cudaFuncAttributeMaxDynamicSharedMemorySize, kRotSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_residual64_cols<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_residual64_cols<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_residual64_cols<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidSmem));
  LAPH_TRY(neglap64_init());
  return small_init();
}
bool gram_splits(long long units) { return units <= kGramSplitUnits; }
int gram(const ProbDesc* pd, const ProbState* ps, const int* start, int np, int nblk, int split, int chunk_rows,
         const double2* W, const double2* Y, double2* gpart, cudaStream_t st) {
  if (split)
    k_gram_split<<<4 * nblk, 128, kGramSplitSmem, st>>>(pd, ps, start, np, chunk_rows, W, Y, gpart);
  else
    k_gram<<<nblk, 64, kGramSmem, st>>>(pd, ps, start, np, chunk_rows, W, Y, gpart);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int gram_reduce(const ProbDesc* pd, const ProbState* ps, const int* start, int np, int nblk, const double2* gpart,
                double2* KK, cudaStream_t st) {
  k_gram_reduce<<<nblk, 256, 0, st>>>(pd, ps, start, np, gpart, KK);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int coef(const ProbDesc* pd, const ProbState* ps, int np, const double* theta, double* tcoef, double* scol, int m,
         const int* dm, cudaStream_t st) {
  k_coef<<<np, 256, 0, st>>>(pd, ps, np, theta, tcoef, scol, m, dm);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int rotate(const ProbDesc* pd, const ProbState* ps, const int* start, int np, int nblk, const double2* W,
           const double2* KK, double2* V, cudaStream_t st) {
  k_rotate<<<nblk, 128, kRotSmem, st>>>(pd, ps, start, np, W, KK, V);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int residual64(const ProbDesc* pd, const ProbState* ps, const int* start, int np, int nblk, const double2* U64,
               const double2* V, const double* theta, float2* S, double* rpart, cudaStream_t st) {
  k_residual64<<<nblk, 128, 0, st>>>(pd, ps, start, np, U64, V, theta, S, rpart);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int residual64_cols(const ProbDesc* pd, const ProbState* ps, const int* start, int np, int nblk, int cols,
                    const double2* U64, const double2* V, const double* theta, float2* S, double* rpart, cudaStream_t st) {
  if (cols >= 4 * kGroups64)
    k_residual64_cols<4><<<nblk, kThreads64, kResidSmem, st>>>(pd, ps, start, np, cols, U64, V, theta, S, rpart);
  else if (cols >= 2 * kGroups64)
    k_residual64_cols<2><<<nblk, kThreads64, kResidSmem, st>>>(pd, ps, start, np, cols, U64, V, theta, S, rpart);
  else
    k_residual64_cols<1><<<nblk, kThreads64, kResidSmem, st>>>(pd, ps, start, np, cols, U64, V, theta, S, rpart);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int resid_check(const ProbDesc* pd, ProbState* ps, int np, const double* rpart, double* resid, double tol,
                int* n_active, cudaStream_t st) {
  k_resid<<<np, 256, 0, st>>>(pd, ps, rpart, resid, tol, n_active);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}
int phase_fix(const ProbDesc* pd, const int* start, int np, int nblk, double2* V, double* phases, double* norms,
              int apply, cudaStream_t st) {
  k_phase_fix<<<nblk, 256, 0, st>>>(pd, start, np, V, phases, norms, apply);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}

}  // namespace laph
