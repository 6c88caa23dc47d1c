// stencil64cols.cuh -- the FP64 block stencil (-Delta) of the Rayleigh-Ritz
// step: a CTA holds the 3 forward and 3 backward links of 128 sites in shared
// memory (110 KB) for a block of columns, and two groups of 128 threads walk
// the block, each thread NC columns of its site per trip; colour-major columns,
// so every warp access is a dense 512-byte segment.
//
// 96 bytes of HBM per site and column at least, but a column also takes 21
// 16-byte loads through L1 and, where links sit in shared memory, their reads:
// latency and the L1 path bound it.  NC = 4 spreads a link read over 4 columns
// and keeps 8 loads of every thread in flight; 2 CTAs of 8 warps fit an SM at 128
// registers.  The links in registers (forward) and shared memory (backward)
// with one column per trip, 12 warps an SM, took 2.75 ms for A W and 2.70 ms
// for the residual at 48^3 x 2 timeslices x 224 columns, this 1.88 and 1.77 ms
// (2.5 and 2.7 TB/s); 24^3 x 6 x 160: 0.74 and 0.71 ms -> 0.49 and 0.47 ms.
// NC = 2: 2.00 and 2.02 ms, NC = 1: 2.36 and 2.65 ms; the bulk prefetch of the
// next trip into L2 gives 5% of it.
#pragma once
#include "batch.cuh"
#include "filter_common.cuh"

namespace laph {

constexpr int kColsFP64 = 32;  // columns per CTA, fewer for small batches (solver.cu)
constexpr int kSites64 = 128;  // sites per CTA
constexpr int kGroups64 = 2;   // thread groups per CTA, each on its own columns
constexpr int kThreads64 = kGroups64 * kSites64;
constexpr int kTrip64 = 4 * kGroups64;  // columns per trip at most
constexpr int kStencil64Smem = 54 * kSites64 * (int)sizeof(double2);  // 110 KB: dynamic, opted in

// The tile's rows of a column (sites s0 ..) into L2.
__device__ __forceinline__ void prefetch64(const double2* x, int V3, int s0) {
#pragma unroll
  for (int c = 0; c < 3; ++c) l2_prefetch(x + (size_t)c * V3 + s0, 16u * min(kSites64, V3 - s0));
}

// Links of the tile's sites into sU (rows 0..26 forward, 27..53 backward
// U_mu(s - mu)): group 0 copies the forward ones, group 1 the backward ones.
__device__ __forceinline__ void load_links64(const double2* __restrict__ U, const Lat& g, int s, const int* dn,
                                             double2 (*sU)[kSites64], int i, int grp) {
#pragma unroll
  for (int mu = 0; mu < 3; ++mu) {
    const int src = grp ? dn[mu] : s;
#pragma unroll
    for (int e = 0; e < 9; ++e) sU[27 * grp + mu * 9 + e][i] = __ldg(U + (size_t)(mu * 9 + e) * g.V3 + src);
  }
}

// hop(x)(s) = sum_mu U_mu(s) x(s+mu) + U_mu(s-mu)^dag x(s-mu) on NC colour-major columns, column c at x + co[c].
template <int NC>
__device__ __forceinline__ void hop64_cols(const double2 (*sU)[kSites64], int i, int V3, const int* up, const int* dn,
                                           const double2* __restrict__ x, const int* co, double2 acc[NC][3]) {
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = acc[c][2] = make_double2(0.0, 0.0);
#pragma unroll
  for (int mu = 0; mu < 3; ++mu)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      double2 xu[NC], xd[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        xu[c] = __ldg(x + co[c] + b * V3 + up[mu]);
        xd[c] = __ldg(x + co[c] + b * V3 + dn[mu]);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double2 uf = sU[mu * 9 + 3 * a + b][i], ub = sU[27 + mu * 9 + 3 * b + a][i];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          cfma(acc[c][a], uf, xu[c]);
          cfmac(acc[c][a], ub, xd[c]);
        }
      }
    }
}

}  // namespace laph
