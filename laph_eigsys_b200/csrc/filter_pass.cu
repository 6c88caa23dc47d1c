// filter_pass.cu -- a whole Chebyshev pass in one kernel, for batches too small
// to keep the step kernels busy.
//
// The step kernels (filter.cu) launch once per step, and a CTA walks 32 columns
// of its sites one after another.  With few site-columns that walk is the time
// of a step whatever the lattice (32 us at 11^3, 64 columns) and most SMs idle.
// Columns do not interact, so here a pass is turned around: a team of CTAs holds
// one lattice, takes a few columns of it, runs all m - 1 steps on them, then
// takes the next few, and as many teams run side by side as fit the chip.  The
// site's links are loaded once per problem (two of the forward directions in 36
// registers, the rest in shared memory) and kept for the pass, X, Z and S of the
// columns in flight stay in L2, and there is one launch per pass instead of one
// conditional node and launch per step.  Between steps the team's CTAs meet at
// a counter (release add, acquire poll); two CTAs of different teams share an
// SM, so one computes while the other waits.
//
// Measured, site-columns per second (step kernels -> this one): 8^3, 64 columns
// 1.2e9 -> 7.0e9; 8^3 x 16, 96 columns 1.9e10 -> 3.8e10; 16^3, 96 columns 0.8e10
// -> 3.4e10; 16^3 x 4 3.0e10 -> 4.1e10; 32^3, 64 columns 3.5e10 -> 4.1e10.  At
// 24^3 x 2, 160 columns (4.4e6 site-columns a step) the step kernels are ahead,
// 4.1e10 (column blocks of 16) against 3.6e10, and at 32^3 x 12 they stream 5.0e10
// (5.0 TB/s of HBM) where this kernel holds 4.1e10: with every access in L2 it is
// bound by load latency at 16 warps per SM and the wait between steps.  Hence
// the line at kPassMaxWork.  (Also measured at 32^3 x 12: all forward links in
// registers 3.7e10, one column at a time 3.5e10, three groups of 224 threads
// sharing one set of links in shared memory 4.6e10, of four 3.1e10.)
//
// The arithmetic per site and column is that of the step kernel, operation for
// operation, so results are the same to the last bit.
#include "filter_pass.cuh"

#include <algorithm>

#include "filter.cuh"
#include "filter_common.cuh"

namespace laph {
namespace {

constexpr int kPassThreads = 256;  // one site each; 2 CTAs of 128 registers a thread per SM
constexpr int kPassCols = 16;      // columns of a team at most
constexpr int kRegDirs = 2;        // directions whose forward links stay in registers
constexpr int kPassSmem = (27 + 9 * (3 - kRegDirs)) * kPassThreads * (int)sizeof(float2);
constexpr long long kPassMaxWork = 3000000;  // site-columns of the batch (all columns, sites) up to which a pass runs here
constexpr int kPassLine = 32;      // ints between two teams' counters (a 128-byte line each)
constexpr unsigned kPassSpin = 1u << 22;  // polls before a wait gives up (a few seconds)

// plan: [kPassClasses][2 + np + 1] (columns per unit, units, prefix of units per problem), then the teams' counters
constexpr int kMaxTeams = 1024;
__host__ __device__ inline size_t plan_stride(int np) { return (size_t)np + 4; }
__host__ __device__ inline size_t plan_ctr(int np) { return (kPassClasses * plan_stride(np) + kPassLine) / kPassLine * kPassLine; }

// One CTA per extent: the unlocked columns of its active problems in units of
// G columns, G as small as gives every team a unit in each of the rounds that
// gmax columns per team would take anyway; and the teams' counters back to zero.
__global__ void __launch_bounds__(256) k_pass_plan(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps,
                                                   int np, PassClass c0, PassClass c1, PassClass c2, PassClass c3,
                                                   int* plan) {
  const PassClass cls[kPassClasses] = {c0, c1, c2, c3};
  const int c = blockIdx.x, tid = threadIdx.x;
  const PassClass g = cls[c];
  int* o = plan + c * plan_stride(np);
  int* ustart = o + 2;
  __shared__ int s_total, s_scan[256];
  if (tid == 0) s_total = 0;
  __syncthreads();
  int cols = 0;
  for (int p = tid; p < np; p += 256)
    if (ps[p].active && pd[p].L == g.L) cols += pd[p].k - ps[p].nlock;
  atomicAdd(&s_total, cols);
  __syncthreads();
  const int rounds = max(1, (s_total + g.teams * g.gmax - 1) / (g.teams * g.gmax));
  const int G = min(g.gmax, max(2, ((s_total + g.teams * rounds - 1) / (g.teams * rounds) + 1) / 2 * 2));
  int base = 0;
  for (int p0 = 0; p0 < np; p0 += 256) {
    const int p = p0 + tid;
    int u = 0;
    if (p < np && ps[p].active && pd[p].L == g.L) u = (pd[p].k - ps[p].nlock + G - 1) / G;
    s_scan[tid] = u;
    __syncthreads();
    for (int d = 1; d < 256; d <<= 1) {
      const int t = tid >= d ? s_scan[tid - d] : 0;
      __syncthreads();
      s_scan[tid] += t;
      __syncthreads();
    }
    if (p < np) ustart[p] = base + s_scan[tid] - u;
    base += s_scan[255];
    __syncthreads();
  }
  if (tid == 0) {
    o[0] = G;
    o[1] = base;
    ustart[np] = base;
  }
  int* ctr = plan + plan_ctr(np) + (size_t)c * kMaxTeams * kPassLine;
  for (int t = tid; t < g.teams; t += 256) ctr[t * kPassLine] = 0;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// All CTAs of a team: every write before the call is visible to every read after
// it.  `target`: the counter's value once all have arrived.  False when the wait
// gave up here or elsewhere; the kernel then returns.
__device__ __forceinline__ bool team_barrier(unsigned* ctr, unsigned target, int* err, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    int ok = 1;
    unsigned it = 0;
    while ((int)(ld_acquire(ctr) - target) < 0)
      if ((++it & 1023u) == 0 && (it > kPassSpin || *reinterpret_cast<volatile int*>(err))) {
        atomicExch(err, 1);
        ok = 0;
        break;
      }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

struct Site {
  int V3, dim, s;       // sites, column stride, own site
  int up[3], dn[3];
};

// One step on the unit's nc columns at this thread's site, two columns at a time: X, Z, S, Y at the first column, cf
// the step's coefficients.  One shared-memory read of a backward link serves both columns.  The neighbour values
// stream through a three-slot register ring, one (direction, colour) of both columns per slot, loaded three slots
// ahead and across the turn to the next pair, so the L2 latency of a load is spent on the slots before it.  An odd
// last column is paired with itself.
struct Slot {
  float2 u[2], d[2];
};

template <bool HAS_S>
__device__ __forceinline__ void pass_step(const Site& t, const float2 (&uf)[kRegDirs][9], const float2 (*sUb)[kPassThreads],
                                          const float2* X, const float2* Z, const float2* __restrict__ S, float2* Y,
                                          const float4* cf, int nc, bool valid) {
  Slot ring[3];
  auto load = [&](Slot& r, const float2* x, unsigned second, int st) {  // slot st = 3 mu + colour
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2* xc = x + (unsigned)((st % 3) * t.V3) + (c ? second : 0u);
      r.u[c] = xc[t.up[st / 3]];
      r.d[c] = xc[t.dn[st / 3]];
    }
  };
  unsigned second = nc > 1 ? t.dim : 0;
#pragma unroll
  for (int st = 0; st < 3; ++st) load(ring[st], X, second, st);
#pragma unroll 1
  for (int j = 0; j < nc; j += 2) {
    const float2* x = X + (unsigned)(j * t.dim);
    const float2* xn = j + 2 < nc ? x + 2 * t.dim : x;  // the next pair (or this one again after the last)
    const unsigned sn = j + 2 < nc && j + 3 >= nc ? 0u : second;
    // packed FP32x2: with u = (re, im), P += (x.re, x.re) u and T += (x.im, x.im) u
    // give u x = (P.x - T.y, P.y + T.x); backward links are stored conjugated
    unsigned long long P[2][3], T[2][3];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int a = 0; a < 3; ++a) P[c][a] = T[c][a] = 0ull;
#pragma unroll
    for (int st = 0; st < 9; ++st) {
      const int mu = st / 3, b = st % 3;
      Slot& v = ring[st % 3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float2 fw = mu < kRegDirs ? uf[mu < kRegDirs ? mu : 0][3 * a + b]
                                        : sUb[27 + (mu - kRegDirs) * 9 + 3 * a + b][threadIdx.x];
        const unsigned long long lf = pk2(fw.x, fw.y);
        const float2 bw = sUb[mu * 9 + 3 * b + a][threadIdx.x];
        const unsigned long long lb = pk2(bw.x, bw.y);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          ffma2(P[c][a], pk2(v.u[c].x, v.u[c].x), lf);
          ffma2(T[c][a], pk2(v.u[c].y, v.u[c].y), lf);
          ffma2(P[c][a], pk2(v.d[c].x, v.d[c].x), lb);
          ffma2(T[c][a], pk2(v.d[c].y, v.d[c].y), lb);
        }
      }
      if (st < 6) load(v, x, second, st + 3);
      else load(v, xn, sn, st - 6);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float4 q = cf[j + c];  // (a c_hop, a c_diag, z, g)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const unsigned o = (unsigned)(j * t.dim + a * t.V3) + (c ? second : 0u);
        const float2 pp = unpk2(P[c][a]), tt = unpk2(T[c][a]);
        const float2 acc = make_float2(pp.x - tt.y, pp.y + tt.x);
        const float2 xs = (X + o)[t.s];
        const float2 ss = HAS_S ? __ldg(S + o + t.s) : make_float2(0.f, 0.f);
        const float2 zz = (Z + o)[t.s];
        float2 r;
        r.x = fmaf(q.z, zz.x, fmaf(q.x, acc.x, fmaf(q.y, xs.x, q.w * ss.x)));
        r.y = fmaf(q.z, zz.y, fmaf(q.x, acc.y, fmaf(q.y, xs.y, q.w * ss.y)));
        if (valid && (c == 0 || second)) (Y + o)[t.s] = r;
      }
    }
    second = sn;
  }
}

template <typename LT>
__global__ void __launch_bounds__(kPassThreads, 2)
    k_cheb_pass(const ProbDesc* __restrict__ pd, const ProbState* __restrict__ ps, int np, PassClass g, int cidx,
                const LT* __restrict__ links, const float* __restrict__ scale, const float2* Sp, float2* E0, float2* E1,
                const double2* Vp, double2* Wp, const double* __restrict__ tcoef, int m, const int* __restrict__ dm,
                int* plan, int* err) {
  extern __shared__ float2 sUb_dyn[];
  float2 (*sUb)[kPassThreads] = reinterpret_cast<float2 (*)[kPassThreads]>(sUb_dyn);
  __shared__ float4 cf[2][kPassCols + 1];
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  if (dm) m = *dm;
  if (*reinterpret_cast<volatile int*>(err)) return;
  const int team = blockIdx.x / g.tiles, tile = blockIdx.x - team * g.tiles;
  const int* o = plan + cidx * plan_stride(np);
  const int G = o[0], nunits = o[1];
  const int* ustart = o + 2;
  unsigned* ctr = reinterpret_cast<unsigned*>(plan) + plan_ctr(np) + ((size_t)cidx * kMaxTeams + team) * kPassLine;
  const Lat lat{g.L, g.L * g.L, g.L * g.L * g.L};
  Site t;
  t.V3 = lat.V3;
  t.dim = 3 * lat.V3;
  // threads past the tile or the lattice compute its last site again and write nothing
  const bool valid = tid < g.ns && tile * g.ns + tid < t.V3;
  t.s = min(tile * g.ns + min(tid, g.ns - 1), t.V3 - 1);
  const bool lane_warp = (tid & ~31) < g.ns;  // warps wholly past the tile only take part in the barriers
  {
    int x, y, z;
    site_xyz(lat, t.s, x, y, z);
#pragma unroll
    for (int mu = 0; mu < 3; ++mu) {
      t.up[mu] = nb_up(lat, x, y, z, mu);
      t.dn[mu] = nb_dn(lat, x, y, z, mu);
    }
  }
  float2* E[2] = {E0 + (size_t)team * g.gmax * t.dim, E1 + (size_t)team * g.gmax * t.dim};
  float2 uf[kRegDirs][9];
  int cur = -1;         // problem whose links are loaded
  int ring = 0;         // E[ring] takes the first step of the next unit
  unsigned target = 0;  // of the team's counter at its next barrier
  for (int u = team; u < nunits; u += g.teams) {
    const int p = find_prob(ustart, np, u);
    const ProbDesc d = pd[p];
    const int j0 = ps[p].nlock + (u - ustart[p]) * G, nc = min(G, d.k - j0);
    const double c_hop = ps[p].c_hop, c_diag = ps[p].c_diag;
    const int direct = ps[p].direct;
    auto coefs = [&](int n) {  // step n's coefficients of this unit's columns
      if (tid < nc) {
        const double* tc = tcoef + d.tc + (size_t)n * 3 * d.k + j0 + tid;
        const double a = tc[0];
        cf[n & 1][LAPH_IX(tid, kPassCols)] =
            make_float4((float)(a * c_hop), (float)(a * c_diag), (float)tc[d.k], (float)tc[2 * d.k]);
      }
    };
    if (p != cur && lane_warp) {
      const LT* U = links + d.uf;
      const float* scl = scale + d.sc;
#pragma unroll
      for (int mu = 0; mu < 3; ++mu)
#pragma unroll
        for (int e = 0; e < 9; ++e) {
          const float2 f = ld_lk(U, scl, (size_t)(mu * 9 + e) * t.V3 + t.s, t.s);
          if (mu < kRegDirs) uf[mu < kRegDirs ? mu : 0][e] = f;
          else sUb[27 + (mu - kRegDirs) * 9 + e][tid] = f;
          float2 b = ld_lk(U, scl, (size_t)(mu * 9 + e) * t.V3 + t.dn[mu], t.dn[mu]);
          b.y = -b.y;  // stored conjugated for the packed hop
          sUb[mu * 9 + e][tid] = b;
        }
    }
    cur = p;
    coefs(1);
    __syncthreads();
    const size_t col = (size_t)d.blk + (size_t)LAPH_IX(j0, d.k) * d.dim;
    const float2* S = Sp + col;
    for (int n = 1; n < m; ++n) {
      float2* Y = E[(n - 1 + ring) & 1];  // its content two steps ago is Z: read and overwritten by its own thread only
      const float2* X = n == 1 ? S : E[(n + ring) & 1];
      const float2* Z = n < 3 ? S : Y;    // steps 1 and 2 have no Z: its coefficient is 0
      if (n < m - 1) coefs(n + 1);
      if (lane_warp) {
        if (n < 3 || !direct) pass_step<true>(t, uf, sUb, X, Z, S, Y, cf[n & 1], nc, valid);
        else pass_step<false>(t, uf, sUb, X, Z, S, Y, cf[n & 1], nc, valid);
      }
      if (n < m - 1) {
        target += g.tiles;
        if (!team_barrier(ctr, target, err, &s_ok)) return;
      }
    }
    if (valid) {  // W = T_m(theta_B) V + E_m in FP64, from this thread's own values
      const float2* Y = E[(m + ring) & 1];
      const double* tm = tcoef + d.tc + (size_t)m * 3 * d.k + j0;
      for (int j = 0; j < nc; ++j)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const size_t i = (size_t)j * t.dim + a * t.V3 + t.s;
          const float2 r = Y[i];
          const double2 v = __ldcs(Vp + col + i);
          const double f = __ldg(tm + j);
          __stcs(Wp + col + i, make_double2(fma(f, v.x, (double)r.x), fma(f, v.y, (double)r.y)));
        }
    }
    // The last step read E[(m - 1 + ring) & 1] of neighbouring tiles, which may still be at it; the other buffer, in
    // which only a site's own Z was read, takes the next unit's first step, and the barrier after that step covers
    // the rest.  The unit's coefficients are replaced only after this CTA is done with them.
    ring = (ring + m) & 1;
    __syncthreads();
  }
  // locked columns: W = V
  const int nthr = (int)gridDim.x * kPassThreads, gt = blockIdx.x * kPassThreads + tid;
  for (int p = 0; p < np; ++p) {
    if (pd[p].L != g.L || !ps[p].active) continue;
    const long long n = (long long)ps[p].nlock * t.dim;
    const double2* v = Vp + pd[p].blk;
    double2* w = Wp + pd[p].blk;
    for (long long i = gt; i < n; i += nthr) __stcs(w + i, __ldg(v + i));
  }
}

}  // namespace

size_t pass_plan_ints(int np) { return plan_ctr(np) + (size_t)kPassClasses * kMaxTeams * kPassLine; }

void PassSize::add(int L, int k) {
  work += (long long)L * L * L * k;
  int c = 0;
  while (c < extents && c < kPassClasses && seen[c] != L) ++c;
  if (c < extents && c < kPassClasses) return;
  if (c < kPassClasses) seen[c] = L;
  extents = c + 1;  // kPassClasses + 1: one too many, and stays so
}
bool PassSize::small() const { return work <= kPassMaxWork && extents <= kPassClasses; }

int pass_layout(const std::vector<ProbDesc>& probs, int bf16, std::vector<PassClass>* out) {
  out->clear();
  PassSize size;
  for (const ProbDesc& d : probs) size.add(d.L, d.k);
  if (!size.small()) return LAPH_OK;
  int dev = 0, sms = 0, occ = 0;
  const void* fn = bf16 ? (const void*)k_cheb_pass<__nv_bfloat162> : (const void*)k_cheb_pass<float2>;
  LAPH_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem));
  LAPH_CUDA_TRY(cudaGetDevice(&dev));
  LAPH_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  LAPH_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kPassThreads, kPassSmem));
  const int slots = sms * occ;
  std::vector<PassClass> cls;
  for (const ProbDesc& d : probs) {
    size_t c = 0;
    while (c < cls.size() && cls[c].L != d.L) ++c;
    if (c == cls.size()) {
      // sites per CTA: the tile whose teams keep the most sites in flight per step time (a step takes as long as a
      // tile has sites, plus about 16 sites' worth of waiting)
      PassClass g{d.L, 0, 0, 0, 0};
      double best = 0.0;
      for (int ns = kPassThreads; ns >= 32; ns -= 32) {
        const int tiles = (d.V3 + ns - 1) / ns, teams = std::min(slots / tiles, kMaxTeams);
        if (teams < 1) break;
        const double v = (double)teams * d.V3 / (ns + 16);
        if (v > best * 1.0001) {
          best = v;
          g.ns = ns;
          g.tiles = tiles;
          g.teams = teams;
        }
      }
      if (g.teams < 1) return LAPH_OK;
      cls.push_back(g);
    }
    cls[c].gmax += d.k;  // columns of the extent, for now
  }
  for (PassClass& g : cls) {
    const int cols = g.gmax;
    g.gmax = std::min(kPassCols, std::max(2, (cols / g.teams + 1) / 2 * 2));
    g.teams = std::max(1, std::min(g.teams, cols / g.gmax));  // the teams' scratch columns fit the extent's own blocks
  }
  *out = cls;
  return LAPH_OK;
}

int filter_pass(const std::vector<PassClass>& cls, const ProbDesc* pd, const ProbState* ps, int np, int bf16,
                const void* links, const float* scale, const float2* S, float2* E0, float2* E1, const double2* V,
                double2* W, const double* tcoef, int m, const int* dm, int* plan, int* err, cudaStream_t st) {
  PassClass c[kPassClasses] = {};
  for (size_t i = 0; i < cls.size(); ++i) c[i] = cls[i];
  k_pass_plan<<<(unsigned)cls.size(), 256, 0, st>>>(pd, ps, np, c[0], c[1], c[2], c[3], plan);
  LAPH_CUDA_TRY(cudaGetLastError());
  for (size_t i = 0; i < cls.size(); ++i) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cls[i].tiles * cls[i].teams);
    cfg.blockDim = dim3(kPassThreads);
    cfg.dynamicSmemBytes = kPassSmem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;  // the teams' CTAs wait on one another
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (bf16)
      LAPH_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_cheb_pass<__nv_bfloat162>, pd, ps, np, cls[i], (int)i,
                                       reinterpret_cast<const __nv_bfloat162*>(links), scale, S, E0, E1, V, W, tcoef, m,
                                       dm, plan, err));
    else
      LAPH_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_cheb_pass<float2>, pd, ps, np, cls[i], (int)i,
                                       reinterpret_cast<const float2*>(links), scale, S, E0, E1, V, W, tcoef, m, dm,
                                       plan, err));
  }
  return LAPH_OK;
}

}  // namespace laph
