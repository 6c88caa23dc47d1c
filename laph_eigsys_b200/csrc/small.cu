// small.cu -- the small dense step of the Rayleigh-Ritz: per problem, from the
// Gram matrices G = W^H W and H = W^H A W (k x k) to the Ritz values and the
// rotation's coefficients C, spread over many CTAs per problem:
//
//   k_project   against the frozen columns [0, c0): G', H' of the active block
//   k_chol      D = diag(G')^-1/2, D G' D = R^H R (blocked, one CTA)
//   k_trinv     X = R^-1, one CTA per 32-row block
//   k_prod<0>   T1 = H' (D X);  k_prod<1>  Ht = (D X)^H T1, its Hermitian part
//   k_jacobi    two-sided Jacobi sweeps of Ht, one thread-block cluster per
//               problem; every rotation goes to a log; Ritz values, order, window
//   k_apply     Q = J_1 J_2 ... from the log, rows independent
//   k_prod<2>   C_a = D X Q
//   k_lift      the rows of C that undo the projection, -G_la C_a
//
// Work matrices per problem (column-major, leading dimension k) at kk, and what
// they hold in turn: [0] G -> R (active block) -> Q, [1] H -> rotations of the
// odd sweeps, [2] X, [3] T1 -> rotations of the even sweeps, [4] Ht -> C.  Columns
// [0, c0) are frozen Ritz vectors: n = k - c0 active columns, and every active
// matrix keeps the leading dimension k.
//
// One CTA of 1024 threads did all of this before and was bound by what one SM
// can move through L2 (the Jacobi alone reads and writes Ht and Q in every one
// of its 2 (n - 1) steps): 11.0 ms per pass at n = 160, 42 ms at n = 256, while
// the rest of the chip idled.  Now the only serial chains are the Jacobi's
// steps (shared memory of a cluster) and the Cholesky's columns; per pass at
// n = 160, us before -> now: Cholesky 1540 -> 165, inverse 906 -> 63, projection
// 1500 -> 43, Jacobi 6380 -> 772, C 537 -> 160.  Every element
// still sees the same operations in the same order as in the unblocked loops
// (sums run over ascending q, updates subtract one term at a time), so the split
// over tiles and CTAs does not change a bit of the result.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "dense.cuh"

namespace cg = cooperative_groups;

namespace laph {
namespace {

constexpr int NB = 32;          // tile of every blocked step (block widths are multiples of it)
constexpr int LDT = NB + 1;     // leading dimension of a staged tile (odd: conflict-free both ways)

struct Small {
  int k, c0, n;
  double2 *G, *H, *X, *T1, *Ht;  // the five work matrices
  double2 *Ga, *Ha;              // active blocks of G and H
  double *dinv, *lam;            // column scaling, Jacobi diagonal by position
  int *perm, *nsteps;            // rank of each position, Jacobi steps in the log
  double* th;                    // Ritz values
};

__device__ __forceinline__ Small small_view(const ProbDesc& d, const ProbState& s, double2* KK, double* theta,
                                            double* dwork) {
  Small v;
  v.k = d.k;
  v.c0 = s.c0;
  v.n = d.k - s.c0;
  const size_t kk2 = (size_t)d.k * d.k;
  v.G = KK + d.kk;
  v.H = v.G + kk2;
  v.X = v.G + 2 * kk2;
  v.T1 = v.G + 3 * kk2;
  v.Ht = v.G + 4 * kk2;
  v.Ga = v.G + v.c0 + (size_t)v.c0 * d.k;
  v.Ha = v.H + v.c0 + (size_t)v.c0 * d.k;
  v.dinv = dwork + d.kv * 4;  // four k-length scratch vectors per problem
  v.lam = v.dinv + d.k;
  v.perm = reinterpret_cast<int*>(v.lam + d.k);
  v.nsteps = reinterpret_cast<int*>(v.lam + 2 * d.k);
  v.th = theta + d.kv;
  return v;
}

// phase boundaries (global timer, ns) for the solver's trace
__device__ __forceinline__ void stamp(unsigned long long* ts, int p, int ph) {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  ts[p * kSmallPhases + ph] = t;
}

// acc(2 x 2 per thread of 256, rows ti + 16 a, columns tj + 16 b) over one staged
// slab of NB rows q, a = sA[q][i], b = sB[q][j], one term at a time in ascending q:
//   ADD acc += a b;  ADDC acc += conj(a) b;  SUB acc -= a b;  SUBC acc -= conj(a) b
// (the last two as the factorisation's own update, product first).  Two 16-byte
// reads per 8 FMAs and thread, one of them shared by 16 lanes: FP64-bound.
// (the FMAs of SUB and of k_apply's rotations are spelled out: their rounding does
// not depend on how a loop is compiled)
enum Term { ADD, ADDC, SUB, SUBC };

template <Term OP>
__device__ __forceinline__ void term(double2& acc, const double2 a, const double2 b) {
  if (OP == ADD) {
    cfma(acc, a, b);
  } else if (OP == ADDC) {
    cfmac(acc, a, b);
  } else if (OP == SUB) {
    acc.x -= fma(a.x, b.x, -(a.y * b.y));
    acc.y -= fma(a.y, b.x, a.x * b.y);
  } else {
    acc.x -= a.x * b.x + a.y * b.y;
    acc.y -= a.x * b.y - a.y * b.x;
  }
}

template <Term OP>
__device__ __forceinline__ void slab_mm(double2 (&acc)[2][2], const double2* sA, int lda, const double2* sB, int ldb,
                                        int ti, int tj) {
#pragma unroll 4
  for (int q = 0; q < NB; ++q) {
    const double2 a0 = sA[q * lda + ti], a1 = sA[q * lda + ti + 16];
    const double2 b0 = sB[q * ldb + tj], b1 = sB[q * ldb + tj + 16];
    term<OP>(acc[0][0], a0, b0);
    term<OP>(acc[0][1], a0, b1);
    term<OP>(acc[1][0], a1, b0);
    term<OP>(acc[1][1], a1, b1);
  }
}

// The same over q in [0, nq) for one 32 x 32 tile, 256
// threads; la(q, i) and lb(q, j) read the operands, A_Q / B_Q: q is the
// operand's contiguous index.  The next slab is read while this one is multiplied.
template <Term OP, bool A_Q, bool B_Q, class LA, class LB>
__device__ __forceinline__ void tile_mm(double2 (&acc)[2][2], int nq, LA la, LB lb, double2* sA, double2* sB) {
  const int t = threadIdx.x, ti = t & 15, tj = t >> 4;
  const int lo = t & 31, hi = t >> 5;  // contiguous / strided index of the staging map (8 rows of 32, 4 times)
  double2 ra[4], rb[4];
  auto fetch = [&](int q0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      ra[e] = A_Q ? la(q0 + lo, hi + 8 * e) : la(q0 + hi + 8 * e, lo);
      rb[e] = B_Q ? lb(q0 + lo, hi + 8 * e) : lb(q0 + hi + 8 * e, lo);
    }
  };
  fetch(0);
  for (int q0 = 0; q0 < nq; q0 += NB) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (A_Q) sA[lo * LDT + hi + 8 * e] = ra[e];
      else sA[(hi + 8 * e) * LDT + lo] = ra[e];
      if (B_Q) sB[lo * LDT + hi + 8 * e] = rb[e];
      else sB[(hi + 8 * e) * LDT + lo] = rb[e];
    }
    __syncthreads();
    if (q0 + NB < nq) fetch(q0 + NB);
    slab_mm<OP>(acc, sA, LDT, sB, LDT, ti, tj);
  }
}

__device__ __forceinline__ void zero_acc(double2 (&acc)[2][2]) {
  acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = make_double2(0.0, 0.0);
}

// -------------------------------------------------------- frozen columns ----
// With G_la = V_l^H W_a and H_la = V_l^H A W_a (Gram tiles of the frozen rows),
// V_l^H V_l = I and V_l^H A V_l = Theta_l,  W_a' = W_a - V_l G_la  has
//   G' = G_aa - G_la^H G_la,
//   H' = H_aa - G_la^H H_la - H_la^H G_la + G_la^H Theta_l G_la.
// One CTA per 32 x 32 tile of the active block, G_la and H_la of its rows and of
// its columns staged 32 frozen rows at a time.
constexpr int kProjSmem = 4 * NB * LDT * (int)sizeof(double2);

__global__ void __launch_bounds__(256) k_project(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                                 double2* KK, double* theta, double* dwork) {
  const int p = blockIdx.y;
  if (!ps[p].active || ps[p].c0 == 0) return;
  const ProbDesc d = pd[p];
  const Small v = small_view(d, ps[p], KK, theta, dwork);
  const int T = v.n / NB;
  const int bi = blockIdx.x % T, bj = blockIdx.x / T;
  if (bj >= T) return;
  extern __shared__ double2 psm[];
  const int k = v.k, tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
  const size_t ci = (size_t)(v.c0 + bi * NB) * k, cj = (size_t)(v.c0 + bj * NB) * k;
  const double2* src[4] = {v.G + ci, v.G + cj, v.H + ci, v.H + cj};
  double2 sg[2][2], sh[2][2];
  zero_acc(sg);
  zero_acc(sh);
  for (int q0 = 0; q0 < v.c0; q0 += NB) {
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int q = tid & 31, c = (tid >> 5) + 8 * e;
        psm[m * NB * LDT + q * LDT + c] = src[m][q0 + q + (size_t)c * k];
      }
    __syncthreads();
    for (int q = 0; q < NB; ++q) {
      const double th = v.th[q0 + q];
      const double2* r = psm + q * LDT;
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const double2 gi = r[ti + 16 * a], gj = r[NB * LDT + tj + 16 * b];
          const double2 hi = r[2 * NB * LDT + ti + 16 * a], hj = r[3 * NB * LDT + tj + 16 * b];
          cfmac(sg[a][b], gi, gj);
          cfmac(sh[a][b], gi, hj);
          cfmac(sh[a][b], hi, gj);
          const double2 t = cmulc(gi, gj);
          sh[a][b] = make_double2(sh[a][b].x - th * t.x, sh[a][b].y - th * t.y);
        }
    }
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const size_t o = LAPH_IX(bi * NB + ti + 16 * a, v.n) + (size_t)LAPH_IX(bj * NB + tj + 16 * b, v.n) * k;
      v.Ga[o] = csub(v.Ga[o], sg[a][b]);
      v.Ha[o] = csub(v.Ha[o], sh[a][b]);
    }
}

// -------------------------------------------------------------- Cholesky ----
// D G' D = R^H R (upper triangle of the active block, in place), D =
// diag(G')^-1/2, right-looking in panels of 32 rows by one CTA of 1024 threads.
// The diagonal block is factored one element per thread with one CTA barrier per
// column; the panel's columns are eliminated one per warp (lane = row, four at a
// time); the trailing tiles go to four groups of 256 threads.  SP: the panel
// R_b,: stays in shared memory for the trailing update (n <= kCholSmemN), else it
// is read back from L2.  A pivot that is not above 1e-28 is clamped there and
// flagged (chol_fail).
constexpr int kCholSmemN = 384;
constexpr int chol_smem(int n, bool sp) {
  return (NB * LDT + 2 * NB + (sp ? NB * (n - NB + 1) : 0)) * (int)sizeof(double2);
}

template <bool SP>
__global__ void __launch_bounds__(1024) k_chol(const ProbDesc* __restrict__ pd, ProbState* __restrict__ ps, double2* KK,
                                               double* theta, double* dwork, unsigned long long* tstamp) {
  const int p = blockIdx.x;
  if (!ps[p].active) return;
  const ProbDesc d = pd[p];
  const Small v = small_view(d, ps[p], KK, theta, dwork);
  const int tid = threadIdx.x, k = v.k, n = v.n;
  if (tid == 0) stamp(tstamp, p, 0);
  extern __shared__ double2 csm[];
  double2* sR = csm;              // [NB][LDT] R_bb
  double2* rowA = sR + NB * LDT;  // [2][NB] the eliminated row
  double2* sP = rowA + 2 * NB;    // [NB][ldp] the panel (SP)
  const int ldp = n - NB + 1;
  __shared__ double s_rinv[NB];
  __shared__ int s_fail;
  if (tid == 0) s_fail = 0;
  for (int i = tid; i < n; i += 1024) {
    const double g = v.Ga[i + (size_t)i * k].x;
    v.dinv[i] = g > 0.0 ? 1.0 / sqrt(g) : 1.0;
  }
  __syncthreads();
  const int grp = tid >> 8, gt = tid & 255;  // four groups of 256 threads, a 32 x 32 tile each
  const int ti = gt & 15, tj = gt >> 4;
  for (int base = 0; base < n; base += NB) {
    const bool first = base == 0;  // the scaling D is applied as each element is first read
    const int lane = tid & 31, warp = tid >> 5;
    {
      const int i = warp, j = lane;
      double2 a = make_double2(0.0, 0.0);
      if (i <= j) {
        a = v.Ga[base + i + (size_t)(base + j) * k];
        if (first) a = cscal(a, v.dinv[i] * v.dinv[j]);
      }
      for (int q = 0; q < NB; ++q) {
        const int b = (q & 1) * NB;
        if (i == q) {
          double piv = __shfl_sync(0xffffffffu, a.x, q);
          if (!(piv > 1e-28)) {
            piv = 1e-28;
            if (j == 0) s_fail = 1;
          }
          const double s = sqrt(piv), r = 1.0 / s;
          a = j == q ? make_double2(s, 0.0) : cscal(a, r);
          rowA[b + j] = a;
          if (j == 0) s_rinv[q] = r;
        }
        __syncthreads();
        if (i > q) term<SUBC>(a, rowA[b + i], rowA[b + j]);
      }
      if (i <= j) v.Ga[base + i + (size_t)(base + j) * k] = a;
      sR[i * LDT + j] = a;
    }
    const int m = n - base - NB, mt = m / NB;
    if (m == 0) break;
    __syncthreads();
    // panel: R_b,: by elimination, lane = row
    double2* Pg = v.Ga + base + (size_t)(base + NB) * k;  // panel rows in G
    for (int cb = warp; cb < m; cb += 128) {
      double2 a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = cb + 32 * u;
        a[u] = c < m ? Pg[lane + (size_t)c * k] : make_double2(0.0, 0.0);
        if (first && c < m) a[u] = cscal(a[u], v.dinv[lane] * v.dinv[NB + c]);
      }
      for (int q = 0; q < NB; ++q) {
        const double r = s_rinv[q];
        const double2 f = sR[q * LDT + lane];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          double2 t = cscal(a[u], r);
          t.x = __shfl_sync(0xffffffffu, t.x, q);
          t.y = __shfl_sync(0xffffffffu, t.y, q);
          if (lane == q) a[u] = t;
          if (lane > q) term<SUBC>(a[u], f, t);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = cb + 32 * u;
        if (c >= m) break;
        if (SP) sP[lane * ldp + c] = a[u];
        Pg[lane + (size_t)c * k] = a[u];
      }
    }
    __syncthreads();
    // trailing update of the upper tiles
    const int nt = mt * (mt + 1) / 2;
    for (int e = grp; e < nt; e += 4) {
      int r = e, bi = 0;
      while (r >= mt - bi) {
        r -= mt - bi;
        ++bi;
      }
      const int bj = bi + r;
      double2 acc[2][2];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int i = NB + bi * NB + ti + 16 * a, j = NB + bj * NB + tj + 16 * b;
          acc[a][b] = v.Ga[base + i + (size_t)(base + j) * k];
          if (first) acc[a][b] = cscal(acc[a][b], v.dinv[i] * v.dinv[j]);
        }
      if (SP) {
        slab_mm<SUBC>(acc, sP + bi * NB, ldp, sP + bj * NB, ldp, ti, tj);
      } else {
        for (int q = 0; q < NB; ++q)
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            const double2 l = Pg[q + (size_t)(bi * NB + ti + 16 * a) * k];
#pragma unroll
            for (int b = 0; b < 2; ++b) term<SUBC>(acc[a][b], l, Pg[q + (size_t)(bj * NB + tj + 16 * b) * k]);
          }
      }
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
          v.Ga[base + NB + LAPH_IX(bi * NB + ti + 16 * a, m) +
               (size_t)(base + NB + LAPH_IX(bj * NB + tj + 16 * b, m)) * k] = acc[a][b];
    }
    __syncthreads();
  }
  if (tid == 0) ps[p].chol_fail = s_fail;
}

// X = R^-1 row by row, X_ij = (delta_ij - sum_{q = i..j-1} X_iq R_qj) / R_jj: one CTA
// per block of 32 rows walks the column blocks, the sum over finished blocks as
// tile products, the last block's recursion with lane = column.
__global__ void __launch_bounds__(256) k_trinv(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                               double2* KK, double* theta, double* dwork, unsigned long long* tstamp) {
  const int p = blockIdx.y;
  if (!ps[p].active) return;
  const Small v = small_view(pd[p], ps[p], KK, theta, dwork);
  const int bi = blockIdx.x, k = v.k;
  if (bi == 0 && threadIdx.x == 0) stamp(tstamp, p, 1);
  if (bi * NB >= v.n) return;
  __shared__ double2 sA[NB * LDT], sB[NB * LDT];
  const int ti = threadIdx.x & 15, tj = threadIdx.x >> 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2* Xi = v.X + bi * NB;  // this block's rows
  for (int bj = bi; bj * NB < v.n; ++bj) {
    const double2* Rj = v.Ga + (size_t)(bj * NB) * k;
    double2 s[2][2];
    zero_acc(s);
    if (bi == bj && ti == tj) s[0][0].x = s[1][1].x = 1.0;
    if (bj > bi)
      tile_mm<SUB, false, true>(
          s, (bj - bi) * NB, [&](int q, int i) { return Xi[i + (size_t)(bi * NB + q) * k]; },
          [&](int q, int j) { return Rj[bi * NB + q + (size_t)j * k]; }, sA, sB);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) sB[(ti + 16 * a) * LDT + tj + 16 * b] = s[a][b];
    for (int e = threadIdx.x; e < NB * NB; e += 256) sA[(e & 31) * LDT + (e >> 5)] = Rj[bj * NB + (e & 31) + (size_t)(e >> 5) * k];
    __syncthreads();
    double2 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = sB[(warp * 4 + u) * LDT + lane];
    const double rl = 1.0 / sA[lane * LDT + lane].x;  // lane's own column
    for (int q = 0; q < NB; ++q) {
      const double2 f = sA[q * LDT + lane];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        double2 t = cscal(x[u], rl);
        t.x = __shfl_sync(0xffffffffu, t.x, q);
        t.y = __shfl_sync(0xffffffffu, t.y, q);
        if (lane == q) x[u] = t;
        if (lane > q) term<SUB>(x[u], t, f);
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) sB[(warp * 4 + u) * LDT + lane] = x[u];
    __syncthreads();
    for (int e = threadIdx.x; e < NB * NB; e += 256)
      Xi[(e & 31) + (size_t)LAPH_IX(bj * NB + (e >> 5), v.n) * k] = sB[(e & 31) * LDT + (e >> 5)];
    __syncthreads();
  }
}

// One CTA per 32 x 32 tile.  OP 0: T1 = H' (D X).  OP 1: Ht = (D X)^H T1, a tile and its
// mirror, of which the Hermitian part is kept.  OP 2: C_a = (D X) Q, below the frozen rows.
template <int OP>
__global__ void __launch_bounds__(256) k_prod(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                              double2* KK, double* theta, double* dwork, int q_in_t1,
                                              unsigned long long* tstamp) {
  const int p = blockIdx.y;
  if (!ps[p].active) return;
  const Small v = small_view(pd[p], ps[p], KK, theta, dwork);
  const int T = v.n / NB, k = v.k;
  const int bi = blockIdx.x % T, bj = blockIdx.x / T;
  if (OP == 0 && blockIdx.x == 0 && threadIdx.x == 0) stamp(tstamp, p, 2);
  if (bj >= T || (OP == 1 && bi > bj)) return;
  __shared__ double2 sA[NB * LDT], sB[NB * LDT];
  const int ti = threadIdx.x & 15, tj = threadIdx.x >> 4;
  double2 acc[2][2], mir[2][2];
  zero_acc(acc);
  if (OP == 0) {
    const double2* Hi = v.Ha + bi * NB;
    const double2* Xj = v.X + (size_t)(bj * NB) * k;
    tile_mm<ADD, false, true>(
        acc, (bj + 1) * NB, [&](int q, int i) { return Hi[i + (size_t)q * k]; },
        [&](int q, int j) { return cscal(Xj[q + (size_t)j * k], v.dinv[q]); }, sA, sB);
  } else if (OP == 1) {
    auto half = [&](double2(&o)[2][2], int r, int c) {
      const double2* Xi = v.X + (size_t)(r * NB) * k;
      const double2* Tj = v.T1 + (size_t)(c * NB) * k;
      tile_mm<ADDC, true, true>(
          o, (r + 1) * NB, [&](int q, int i) { return cscal(Xi[q + (size_t)i * k], v.dinv[q]); },
          [&](int q, int j) { return Tj[q + (size_t)j * k]; }, sA, sB);
    };
    half(acc, bi, bj);
    zero_acc(mir);
    if (bi != bj) half(mir, bj, bi);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) sB[(ti + 16 * a) * LDT + tj + 16 * b] = bi == bj ? acc[a][b] : mir[a][b];
    __syncthreads();
  } else {
    const double2* Xi = v.X + bi * NB + (size_t)(bi * NB) * k;
    const double2* Qj = (q_in_t1 ? v.T1 : v.Ga) + bi * NB + (size_t)(bj * NB) * k;
    const double* di = v.dinv + bi * NB;
    tile_mm<ADD, false, true>(
        acc, v.n - bi * NB, [&](int q, int i) { return cscal(Xi[i + (size_t)q * k], di[i]); },
        [&](int q, int j) { return Qj[q + (size_t)j * k]; }, sA, sB);
  }
  double2* O = OP == 0 ? v.T1 : OP == 1 ? v.Ht : v.Ht + v.c0 + (size_t)v.c0 * k;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int i = LAPH_IX(bi * NB + ti + 16 * a, v.n), j = LAPH_IX(bj * NB + tj + 16 * b, v.n);
      double2 r = acc[a][b];
      if (OP == 1) {
        if (i > j) continue;
        if (i == j) {
          r.y = 0.0;
        } else {
          const double2 t = sB[(tj + 16 * b) * LDT + ti + 16 * a];  // Ht(j, i)
          r = make_double2(0.5 * (r.x + t.x), 0.5 * (r.y - t.y));
          O[j + (size_t)i * k] = cconj(r);
        }
      }
      O[i + (size_t)j * k] = r;
    }
}

// ---------------------------------------------------------------- Jacobi ----
// Two-sided cyclic Jacobi in "position order": in every step position i is
// paired with its mirror n-1-i, and after the rotations positions 1..n-1 shift
// by one (round-robin tournament: every pair meets once in n-1 steps).  One
// cluster of C CTAs per problem; CTA c owns the position pairs
// r in [c n/(2C), (c+1) n/(2C)), i.e. columns r and n-1-r, in its shared memory
// (SM), two copies: a step reads one and writes the rotated 2 x 2 blocks to
// their shifted rows and columns in the other.  Only the outermost column pair
// of a CTA moves to a neighbour (distributed shared memory stores).  Each CTA
// computes all n/2 rotations of a step itself, from the owners' diagonal entries
// (three distributed shared memory reads per pair), so a step has one cluster
// barrier and one CTA barrier.  The product of the rotations is not kept here:
// they go to a log that k_apply replays.  n > kJacSmemN16, or a cluster the
// device has no room for, keeps both copies in global memory (Ht and the
// Cholesky factor's storage), same code.
// A step costs 1.4-3.9 us (n = 64 .. 320) where one SM took 4.3-50 us; much of it is
// the chain of square roots and divisions of a rotation.  The test for a rotation needs
// no square root of its own, and up to n = 128 and in global memory (SPLIT) one half
// of the threads takes the chain for the angles, the other for the phases.  Above, the
// second read of every pivot from its owner costs more than that gives (n = 224 1519
// -> 1570, 320 2380 -> 2850).  Clusters of 8 keep to 64 registers, two CTAs an SM: at
// 121 the clusters of 16 problems do not fit the device at once (n = 96 437 -> 673 us).
// 2 sweeps, us, before -> now, 1 or 2 problems: n = 32 115 -> 88, 128 583 -> 552, 160 835
// -> 772, 224 1617 -> 1519, 320 2466 -> 2379, 416 5600 -> 4460; 8 of 64 232 -> 184; 16
// of 64 257 -> 225, of 96 452 -> 437, of 128 692 -> 694, of 160 1010 -> 1001.  Clusters of
// 1, 2 and 4 where they hold the matrix: n = 32 89, 92, 92; 64 290, 231, 206; 160 in 4 1109.
constexpr int kJacThreads = 512;
constexpr int kJacSplitN = 128;  // up to here angles and phases of the rotations run on separate threads
constexpr int kJacSmemN8 = 224, kJacSmemN16 = 320;  // largest n whose two copies fit 8 / 16 CTAs

__device__ __forceinline__ int jac_shift(int pos, int n) { return pos == 0 ? 0 : (pos == n - 1 ? 1 : pos + 1); }

// rr > 1e-300 and rr > 1e-18 sqrt(|app aqq|); the square root only where the squares, a factor 2 apart, do not decide
__device__ __forceinline__ bool jac_rotates(double rr, double app, double aqq) {
  const double m = fabs(app * aqq);
  if (rr > 1e-120 && rr < 1e120 && m < 1e240) {
    const double q = rr * rr;
    if (q > 2e-36 * m) return true;
    if (q < 0.5e-36 * m) return false;
  }
  return rr > 1e-300 && rr > 1e-18 * sqrt(m);
}

template <int C, bool SM, bool SPLIT>
__global__ void __launch_bounds__(kJacThreads, C == 8 ? 2 : 1) k_jacobi(const ProbDesc* __restrict__ pd, ProbState* __restrict__ ps,
                                                        double2* KK, double* theta, double* dwork, int first_iter,
                                                        int fixed_cut, int sweeps, int last,
                                                        unsigned long long* tstamp) {
  const int p = blockIdx.x / C;
  if (!ps[p].active) return;  // the whole cluster
  const Small v = small_view(pd[p], ps[p], KK, theta, dwork);
  cg::cluster_group cl = cg::this_cluster();
  const int rk = (int)cl.block_rank(), tid = threadIdx.x;
  if (rk == 0 && tid == 0) stamp(tstamp, p, 3);
  const int n = v.n, k = v.k, half = n / 2, PP = half / C;
  extern __shared__ double2 jsm[];  // SM: [2][2 PP][n]
  __shared__ double s_c[256], s_s[256];
  __shared__ double2 s_e[256];
  __shared__ double2* s_src[2][64];  // this CTA's columns (pair l: l and PP + l) in either copy ...
  __shared__ double2* s_dst[2][64];  // ... and where each goes
  __shared__ double s_part[2], s_red[2][kJacThreads / 32];
  // column `pos` of copy b, wherever it lives
  auto column = [&](int b, int pos) -> double2* {
    if (!SM) return (b == 0 ? v.Ht : v.Ga) + (size_t)LAPH_IX(pos, n) * k;
    const int r = pos < half ? pos : n - 1 - pos;
    const int col = (pos < half ? 0 : PP) + r % PP;
    return cl.map_shared_rank(jsm, r / PP) + (size_t)(b * 2 * PP + LAPH_IX(col, 2 * PP)) * n;
  };
  auto own_pos = [&](int c) { return c < PP ? rk * PP + c : n - 1 - (rk * PP + c - PP); };
  for (int e = tid; e < 4 * PP; e += kJacThreads) {
    const int b = e / (2 * PP), c = e - b * 2 * PP, pos = own_pos(c);
    s_src[b][c] = SM ? jsm + (size_t)(b * 2 * PP + c) * n : column(b, pos);
    s_dst[b][c] = column(b, jac_shift(pos, n));
  }
  if (SM)
    for (int e = tid; e < 2 * PP * n; e += kJacThreads) {
      const int c = e / n, i = e - c * n;
      jsm[(size_t)c * n + i] = v.Ht[i + (size_t)own_pos(c) * k];
    }
  __syncthreads();
  cl.sync();
  const int pr = SPLIT ? tid & 255 : tid;
  const bool angle = !SPLIT || tid < 256, phase = !SPLIT || tid >= 256, logs = pr / PP == rk;
  // columns of the thread's pair in either copy
  const int pc = min(pr, half - 1);
  const double2 *cp0 = column(0, pc), *cp1 = column(1, pc), *cq0 = column(0, n - 1 - pc), *cq1 = column(1, n - 1 - pc);
  int cur = 0, t = 0;
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int e = tid; e < 2 * PP * n; e += kJacThreads) {
      const int c = e / n, i = e - c * n;
      const double2 x = s_src[cur][c][i];
      if (i != own_pos(c)) off += x.x * x.x + x.y * x.y;
      else dia += x.x * x.x;
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dia += __shfl_xor_sync(0xffffffffu, dia, o);
    }
    if ((tid & 31) == 0) {
      s_red[0][tid >> 5] = off;
      s_red[1][tid >> 5] = dia;
    }
    __syncthreads();
    if (tid < 2) {
      double s = 0.0;
      for (int w = 0; w < kJacThreads / 32; ++w) s += s_red[tid][w];
      s_part[tid] = s;
    }
    cl.sync();
    double so = 0.0, sd = 0.0;  // the same sums in the same order in every CTA
    for (int c = 0; c < C; ++c) {
      const double* q = cl.map_shared_rank(s_part, c);
      so += q[0];
      sd += q[1];
    }
    cl.sync();
    // |off| <= 3e-14 |diag|: with eigenvalue gaps >= 1e-3 lambda_max this
    // leaves eigenvector errors below 1e-10, far under the residual target
    if (so <= 1e-27 * sd) break;
    double2* log = sweep == 0 ? v.H : v.T1;
    for (int step = 0; step < n - 1; ++step, ++t) {
      // rotation of pair r = (r, n-1-r): J (p,p)=c (p,q)=s (q,p)=-s e (q,q)=c e, e = e^{-i phi}
      if (pr < half) {
        const double2 *cp = cur ? cp1 : cp0, *cq = cur ? cq1 : cq0;
        const double2 g = cq[pr];
        const double app = cp[pr].x, aqq = cq[n - 1 - pr].x;
        const double rr = hypot(g.x, g.y);
        const bool rot = jac_rotates(rr, app, aqq);
        double2* o = log + 2 * ((size_t)step * half + pr);
        if (phase) {
          double2 em = make_double2(1.0, 0.0);
          if (rot) em = make_double2(g.x / rr, -g.y / rr);
          s_e[pr] = em;
          if (logs) o[1] = em;
        }
        if (angle) {
          double c = 1.0, s = 0.0;
          if (rot) {
            const double tau = (aqq - app) / (2.0 * rr);
            const double tt = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + tt * tt);
            s = tt * c;
          }
          s_c[pr] = c;
          s_s[pr] = s;
          if (logs) o[0] = make_double2(c, s);
        }
      }
      __syncthreads();
      // Ht <- J^H Ht J on every 2x2 block (rows r', n-1-r'; columns r, n-1-r), shifted
      const int nxt = cur ^ 1;
      for (int e = tid; e < half * PP; e += kJacThreads) {
        const int l = e / half, rp = e - l * half, r = rk * PP + l;
        const int pp = rp, qq = n - 1 - rp;
        const double c = s_c[r], s = s_s[r];
        const double2 em = s_e[r];
        const double c2 = s_c[rp], s2 = s_s[rp];
        const double2 ep = cconj(s_e[rp]);
        const double2 *hp = s_src[cur][l], *hq = s_src[cur][PP + l];
        const double2 a_pp = hp[pp], a_qp = hp[qq], a_pq = hq[pp], a_qq = hq[qq];
        // columns: X = A J
        const double2 t1 = cmul(a_pq, em), t2 = cmul(a_qq, em);
        const double2 x_pp = make_double2(c * a_pp.x - s * t1.x, c * a_pp.y - s * t1.y);
        const double2 x_qp = make_double2(c * a_qp.x - s * t2.x, c * a_qp.y - s * t2.y);
        const double2 x_pq = make_double2(s * a_pp.x + c * t1.x, s * a_pp.y + c * t1.y);
        const double2 x_qq = make_double2(s * a_qp.x + c * t2.x, s * a_qp.y + c * t2.y);
        // rows: B = J'^H X, J'^H (p',p')=c' (p',q')=-s' conj(e') (q',p')=s' (q',q')=c' conj(e')
        const double2 u1 = cmul(x_qp, ep), u2 = cmul(x_qq, ep);
        double2 b_pp = make_double2(c2 * x_pp.x - s2 * u1.x, c2 * x_pp.y - s2 * u1.y);
        double2 b_qp = make_double2(s2 * x_pp.x + c2 * u1.x, s2 * x_pp.y + c2 * u1.y);
        double2 b_pq = make_double2(c2 * x_pq.x - s2 * u2.x, c2 * x_pq.y - s2 * u2.y);
        double2 b_qq = make_double2(s2 * x_pq.x + c2 * u2.x, s2 * x_pq.y + c2 * u2.y);
        if (rp == r) {
          // diagonal block: the rotated pair is decoupled exactly
          if (s != 0.0) b_pq = b_qp = make_double2(0.0, 0.0);
          b_pp.y = 0.0;
          b_qq.y = 0.0;
        }
        double2 *op = s_dst[nxt][l], *oq = s_dst[nxt][PP + l];
        const int npp = LAPH_IX(jac_shift(pp, n), n), nqq = LAPH_IX(jac_shift(qq, n), n);
        op[npp] = b_pp;
        op[nqq] = b_qp;
        oq[npp] = b_pq;
        oq[nqq] = b_qq;
      }
      cl.sync();
      cur = nxt;
    }
  }
  // the diagonal by position, and the matrix itself where more sweeps follow
  for (int c = tid; c < 2 * PP; c += kJacThreads) v.lam[own_pos(c)] = s_src[cur][c][own_pos(c)].x;
  if (!last && (SM || cur == 1))
    for (int e = tid; e < 2 * PP * n; e += kJacThreads) {
      const int c = e / n, i = e - c * n;
      v.Ht[i + (size_t)own_pos(c) * k] = s_src[cur][c][i];
    }
  if (rk == 0 && tid == 0) *v.nsteps = t;
  cl.sync();  // lam complete; no CTA leaves while its shared memory may still be read
  if (rk != 0 || !last) return;
  // rank sort, ties by position
  for (int i = tid; i < n; i += kJacThreads) {
    const double li = v.lam[i];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double lj = v.lam[j];
      r += (lj < li) || (lj == li && j < i);
    }
    v.perm[i] = r;
    v.th[v.c0 + LAPH_IX(r, n)] = li;
  }
  __syncthreads();
  // next window [lam_cut, lam_max]
  if (tid == 0) {
    ProbState& S = ps[p];
    double cut = v.th[k - 1];
    if (fixed_cut || (first_iter && S.lam_cut > 0.0)) cut = S.lam_cut;
    if (cut >= S.lam_max - 1e-3) cut = S.lam_max - 1e-3;
    if (cut < 1e-6) cut = 1e-6;
    S.lam_cut = cut;
    const double al = 2.0 / (S.lam_max - cut);
    S.c_hop = al;
    S.c_diag = (S.lam_max + cut - 12.0) / (S.lam_max - cut);
    S.theta_min = v.th[0];
  }
}

// The logged rotations on the rows of the identity: Q = J_1 J_2 ..., in Ritz order.
// Rows are independent: 16 lanes hold a row in registers, M = n / 32 position
// pairs per lane, so the tournament's shift is a register move plus one shuffle
// each way per step, and only the step's rotations are read, through a
// cp.async ring of kApplyU steps per stage shared by the CTA's four rows.
// FP64- and latency-bound (0.2-0.4 us per step, n = 64 .. 256).
constexpr int kApplyThreads = 64, kApplyRows = kApplyThreads / 16, kApplyU = 4;
// a b, and the two columns of a plane rotation: c x - s y, s x + c y
__device__ __forceinline__ double2 cmul_f(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 rot_p(double c, double s, double2 x, double2 y) {
  return make_double2(fma(c, x.x, -(s * y.x)), fma(c, x.y, -(s * y.y)));
}
__device__ __forceinline__ double2 rot_q(double c, double s, double2 x, double2 y) {
  return make_double2(fma(s, x.x, c * y.x), fma(s, x.y, c * y.y));
}
constexpr int apply_smem(int k) { return 2 * kApplyU * (k / 2) * 2 * (int)sizeof(double2); }

template <int M>
__device__ __forceinline__ void apply_rows(const Small& v, double2* Q, int row, int first, int last, double2* ring) {
  constexpr int n = 32 * M, half = 16 * M;
  const int lane = threadIdx.x & 15, k = v.k;
  const unsigned mask = 0xffffffffu;
  double2 xp[M], xq[M];
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int p = lane * M + i, q = n - 1 - p;
    xp[i] = first ? make_double2(p == row ? 1.0 : 0.0, 0.0) : Q[row + (size_t)p * k];
    xq[i] = first ? make_double2(q == row ? 1.0 : 0.0, 0.0) : Q[row + (size_t)q * k];
  }
  const int nsteps = *v.nsteps;
  auto load = [&](int s) {  // steps [s, s + kApplyU) into their stage of the ring
    double2* st = ring + ((s / kApplyU) & 1) * (kApplyU * half * 2);
    for (int e = threadIdx.x; e < kApplyU * half * 2; e += kApplyThreads) {
      const int u = e / (half * 2), w = e - u * half * 2, t = s + u;
      if (t >= nsteps) break;
      const double2* log = t < n - 1 ? v.H + 2 * (size_t)t * half : v.T1 + 2 * (size_t)(t - (n - 1)) * half;
      // [u][(c, s) | e][pair of the lane][lane]: consecutive lanes read consecutive 16 bytes
      const int r = w >> 1;
      cp_async16(st + ((2 * u + (w & 1)) * M + r % M) * 16 + r / M, log + w, true);
    }
    cp_async_commit();
  };
  load(0);
  for (int s = 0; s < nsteps; s += kApplyU) {
    if (s + kApplyU < nsteps) load(s + kApplyU);
    else cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const double2* st = ring + ((s / kApplyU) & 1) * (kApplyU * half * 2);
    const int nu = min(kApplyU, nsteps - s);
    for (int u = 0; u < nu; ++u) {
      const double2* rot = st + u * half * 2 + lane;
#pragma unroll
      for (int i = 0; i < M; ++i) {
        const double2 cs = rot[16 * i];
        const double2 y = cmul_f(xq[i], rot[16 * (M + i)]), x = xp[i];
        xp[i] = rot_p(cs.x, cs.y, x, y);
        xq[i] = rot_q(cs.x, cs.y, x, y);
      }
      // shift: pair d's p from pair d-1's p (pair 1's from pair 0's q, pair 0's stays), its q from
      // pair d+1's q (the innermost pair's from its own p)
      const double2 q0 = xq[0], pl = xp[M - 1];
      double2 up = M == 1 && lane == 0 ? q0 : pl;
      up.x = __shfl_up_sync(mask, up.x, 1, 16);
      up.y = __shfl_up_sync(mask, up.y, 1, 16);
      double2 dn;
      dn.x = __shfl_down_sync(mask, q0.x, 1, 16);
      dn.y = __shfl_down_sync(mask, q0.y, 1, 16);
      const double2 p0 = xp[0];
#pragma unroll
      for (int i = M - 1; i > 0; --i) xp[i] = xp[i - 1];
      xp[0] = lane == 0 ? p0 : up;
      if (M > 1 && lane == 0) xp[M > 1 ? 1 : 0] = q0;
#pragma unroll
      for (int i = 0; i + 1 < M; ++i) xq[i] = xq[i + 1];
      xq[M - 1] = lane == 15 ? pl : dn;
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  // The row is in registers, so it can go back in place: Ritz order at the end, else position order.  A launch without a
  // step comes here with nothing else between the lanes' reads and their permuted writes.
  __syncwarp();
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int p = lane * M + i, q = n - 1 - p;
    Q[row + (size_t)(last ? LAPH_IX(v.perm[p], n) : p) * k] = xp[i];
    Q[row + (size_t)(last ? LAPH_IX(v.perm[q], n) : q) * k] = xq[i];
  }
}

// MMAX: the widest block of the batch is at most 32 MMAX (the registers of the wide ones stay out of the others).
template <int MMAX>
__global__ void __launch_bounds__(kApplyThreads) k_apply(const ProbDesc* __restrict__ pd,
                                                         const ProbState* __restrict__ ps, double2* KK, double* theta,
                                                         double* dwork, int first, int last, int q_in_t1,
                                                         unsigned long long* tstamp) {
  const int p = blockIdx.y;
  if (!ps[p].active) return;
  const Small v = small_view(pd[p], ps[p], KK, theta, dwork);
  if (blockIdx.x == 0 && threadIdx.x == 0) stamp(tstamp, p, 4);
  if ((int)blockIdx.x * kApplyRows >= v.n) return;
  extern __shared__ double2 rsm[];
  const int row = blockIdx.x * kApplyRows + (threadIdx.x >> 4);
  const int m = v.n / 32;
#define LAPH_APPLY(M) \
  if constexpr (M <= MMAX) if (m == M) return apply_rows<M>(v, q_in_t1 ? v.T1 : v.Ga, row, first, last, rsm);
  LAPH_APPLY(1)
  LAPH_APPLY(2)
  LAPH_APPLY(3)
  LAPH_APPLY(4)
  LAPH_APPLY(5)
  LAPH_APPLY(6)
  LAPH_APPLY(7)
  LAPH_APPLY(8)
  LAPH_APPLY(9)
  LAPH_APPLY(10)
  LAPH_APPLY(11)
  LAPH_APPLY(12)
  LAPH_APPLY(13)
  LAPH_APPLY(14)
  LAPH_APPLY(15)
  LAPH_APPLY(16)
#undef LAPH_APPLY
}

// Rows [0, c0) of the rotation's coefficients: -G_la C_a (they undo the projection).
__global__ void __launch_bounds__(256) k_lift(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                              double2* KK, double* theta, double* dwork, unsigned long long* tstamp) {
  const int p = blockIdx.y;
  if (!ps[p].active) return;
  const Small v = small_view(pd[p], ps[p], KK, theta, dwork);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    stamp(tstamp, p, 5);
    stamp(tstamp, p, 6);
  }
  const int T = v.n / NB, k = v.k;
  const int bj = blockIdx.x % T, bi = blockIdx.x / T;
  if (bi * NB >= v.c0) return;
  __shared__ double2 sA[NB * LDT], sB[NB * LDT];
  double2 acc[2][2];
  zero_acc(acc);
  const double2* Gi = v.G + bi * NB + (size_t)v.c0 * k;
  const double2* Cj = v.Ht + v.c0 + (size_t)(v.c0 + bj * NB) * k;
  tile_mm<ADD, false, true>(
      acc, v.n, [&](int q, int i) { return Gi[i + (size_t)q * k]; },
      [&](int q, int j) { return Cj[q + (size_t)j * k]; }, sA, sB);
  const int ti = threadIdx.x & 15, tj = threadIdx.x >> 4;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      v.Ht[LAPH_IX(bi * NB + ti + 16 * a, v.c0) + (size_t)(v.c0 + LAPH_IX(bj * NB + tj + 16 * b, v.n)) * k] =
          make_double2(-acc[a][b].x, -acc[a][b].y);
}

template <int C, bool SM, bool SPLIT>
int launch_jacobi(const ProbDesc* pd, ProbState* ps, int np, int smem, double2* KK, double* theta, double* dwork,
                  int first_iter, int fixed_cut, int sweeps, int last, unsigned long long* tstamp, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(np * C);
  cfg.blockDim = dim3(kJacThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = C;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  LAPH_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_jacobi<C, SM, SPLIT>, pd, ps, KK, theta, dwork, first_iter, fixed_cut, sweeps, last,
                                   tstamp));
  return LAPH_OK;
}

}  // namespace

int small_init() {
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_project, cudaFuncAttributeMaxDynamicSharedMemorySize, kProjSmem));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_chol<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     chol_smem(kCholSmemN, true)));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_apply<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem(160)));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_apply<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem(256)));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_apply<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, apply_smem(512)));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_jacobi<8, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     4 * kJacSplitN * kJacSplitN));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_jacobi<8, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     4 * kJacSmemN8 * kJacSmemN8));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_jacobi<16, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     2 * kJacSmemN16 * kJacSmemN16));
  LAPH_CUDA_TRY(cudaFuncSetAttribute(k_jacobi<16, true, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return LAPH_OK;
}

// A cluster of 16 CTAs of up to 215 KB, or of 8 of up to 210 KB, may have no room on the device (fewer SMs in every GPC,
// as in a partitioned one); its blocks then take the global-memory form.  Asked once per device: the two questions take
// 0.4 ms, a tenth of creating a small solver.
int small_jacobi_width(int* n) {
  static std::mutex mu;
  static int width[64];
  static bool known[64];
  int dev = 0;
  LAPH_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && known[dev]) {
    *n = width[dev];
    return LAPH_OK;
  }
  auto fits = [](const void* fn, int c, int smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kJacThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return clusters > 0;
  };
  *n = !fits((const void*)k_jacobi<8, true, false>, 8, 4 * kJacSmemN8 * kJacSmemN8)       ? 0
       : !fits((const void*)k_jacobi<16, true, false>, 16, 2 * kJacSmemN16 * kJacSmemN16) ? kJacSmemN8
                                                                                          : kJacSmemN16;
  if (dev < 64) {
    width[dev] = *n;
    known[dev] = true;
  }
  return LAPH_OK;
}

// Problems of one launch: they are grid rows, of which there are 65535 at most.
constexpr int kSmallMaxProbs = 65535;

int small_launches(int np, int kmax, int smem_n, int max_sweeps) {
  const int per = kmax > smem_n ? 1 : 2, groups = (np + kSmallMaxProbs - 1) / kSmallMaxProbs;
  return groups * (7 + 2 * ((max_sweeps + per - 1) / per));
}

int small_dense(const ProbDesc* pd, ProbState* ps, int np, int kmax, int smem_n, double2* KK, double* theta, double* dwork,
                int first_iter, int fixed_cut, int max_sweeps, unsigned long long* tstamp, cudaStream_t st) {
  if (np > kSmallMaxProbs) {
    LAPH_TRY(small_dense(pd + kSmallMaxProbs, ps + kSmallMaxProbs, np - kSmallMaxProbs, kmax, smem_n, KK, theta, dwork,
                         first_iter, fixed_cut, max_sweeps, tstamp + (size_t)kSmallMaxProbs * kSmallPhases, st));
    np = kSmallMaxProbs;
  }
  const int T = kmax / NB;
  const dim3 tiles(T * T, np);
  k_project<<<tiles, 256, kProjSmem, st>>>(pd, ps, KK, theta, dwork);
  if (kmax <= kCholSmemN)
    k_chol<true><<<np, 1024, chol_smem(kmax, true), st>>>(pd, ps, KK, theta, dwork, tstamp);
  else
    k_chol<false><<<np, 1024, chol_smem(kmax, false), st>>>(pd, ps, KK, theta, dwork, tstamp);
  k_trinv<<<dim3(T, np), 256, 0, st>>>(pd, ps, KK, theta, dwork, tstamp);
  k_prod<0><<<tiles, 256, 0, st>>>(pd, ps, KK, theta, dwork, 0, tstamp);
  k_prod<1><<<tiles, 256, 0, st>>>(pd, ps, KK, theta, dwork, 0, tstamp);
  LAPH_CUDA_TRY(cudaGetLastError());
  // The log holds two sweeps, or one where the Jacobi's second copy takes the Cholesky factor's storage and Q
  // the second sweep's log: more sweeps run as further launches on the rotated matrix.
  const int global = kmax > smem_n, per = global ? 1 : 2;
  for (int s = 0; s < max_sweeps; s += per) {
    const int ns = std::min(per, max_sweeps - s), last = s + per >= max_sweeps;
    if (global)
      LAPH_TRY((launch_jacobi<8, false, true>(pd, ps, np, 0, KK, theta, dwork, first_iter, fixed_cut, ns, last, tstamp, st)));
    else if (kmax <= kJacSplitN)
      LAPH_TRY((launch_jacobi<8, true, true>(pd, ps, np, 4 * kmax * kmax, KK, theta, dwork, first_iter, fixed_cut, ns,
                                             last, tstamp, st)));
    else if (kmax <= kJacSmemN8)
      LAPH_TRY((launch_jacobi<8, true, false>(pd, ps, np, 4 * kmax * kmax, KK, theta, dwork, first_iter, fixed_cut, ns, last,
                                       tstamp, st)));
    else
      LAPH_TRY((launch_jacobi<16, true, false>(pd, ps, np, 2 * kmax * kmax, KK, theta, dwork, first_iter, fixed_cut, ns, last,
                                        tstamp, st)));
    const dim3 rows((kmax + kApplyRows - 1) / kApplyRows, np);
    auto apply = kmax <= 160 ? k_apply<5> : kmax <= 256 ? k_apply<8> : k_apply<16>;
    apply<<<rows, kApplyThreads, apply_smem(kmax), st>>>(pd, ps, KK, theta, dwork, s == 0, last, global, tstamp);
  }
  k_prod<2><<<tiles, 256, 0, st>>>(pd, ps, KK, theta, dwork, global, tstamp);
  k_lift<<<tiles, 256, 0, st>>>(pd, ps, KK, theta, dwork, tstamp);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}

}  // namespace laph
