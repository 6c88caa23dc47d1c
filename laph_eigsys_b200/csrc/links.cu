// links.cu -- boundary link layouts and plaquette reductions.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "links.cuh"
#include "su3.cuh"

namespace laph {

int check_links_finite(const double* in, int layout, int V3, const char* who) {
  if (layout != LAPH_LAYOUT_ROWMAJOR && layout != LAPH_LAYOUT_EIGEN && layout != LAPH_LAYOUT_CONF) {
    set_error("%s: unknown link layout %d", who, layout);
    return LAPH_EINVAL;
  }
  // per site: 54 contiguous doubles (ROWMAJOR, EIGEN), or slots 1..3 of 72 (CONF)
  const size_t stride = layout == LAPH_LAYOUT_CONF ? 72 : 54, first = layout == LAPH_LAYOUT_CONF ? 18 : 0;
  long long bad = V3;
#pragma omp parallel for reduction(min : bad) schedule(static)
  for (long long s = 0; s < V3; ++s) {
    const double* p = in + (size_t)s * stride + first;
    bool ok = true;
    for (int e = 0; e < 54; ++e) ok &= std::isfinite(p[e]);
    if (!ok && s < bad) bad = s;
  }
  if (bad < V3) {
    set_error("%s: non-finite link value at site %lld", who, bad);
    return LAPH_EINVAL;
  }
  return LAPH_OK;
}

// sites below this are copied by the calling thread (a parallel region costs more)
constexpr long long kParallelSites = 512;

long long links_pack(const double* in, int layout, long long s0, long long n, double* out) {
  const size_t stride = layout == LAPH_LAYOUT_CONF ? 72 : 54, first = layout == LAPH_LAYOUT_CONF ? 18 : 0;
  long long bad = -1;
  long long lowest = s0 + n;
#pragma omp parallel for reduction(min : lowest) schedule(static) if (n >= kParallelSites)
  for (long long i = 0; i < n; ++i) {
    const double* p = in + (size_t)(s0 + i) * stride + first;
    double* q = out + (size_t)i * 54;
    bool ok = true;
    for (int e = 0; e < 54; ++e) {
      ok &= std::isfinite(p[e]);
      q[e] = p[e];
    }
    if (!ok && s0 + i < lowest) lowest = s0 + i;
  }
  if (lowest < s0 + n) bad = lowest;
  return bad;
}

void links_unpack(const double* in, int layout, long long s0, long long n, double* out) {
  const size_t stride = layout == LAPH_LAYOUT_CONF ? 72 : 54, first = layout == LAPH_LAYOUT_CONF ? 18 : 0;
#pragma omp parallel for schedule(static) if (n >= kParallelSites)
  for (long long i = 0; i < n; ++i) {
    double* q = out + (size_t)(s0 + i) * stride;
    // the temporal slot is not held on the device: the identity goes there
    for (size_t k = 0; k < first; ++k) q[k] = k == 0 || k == 8 || k == 16 ? 1.0 : 0.0;
    std::memcpy(q + first, in + (size_t)i * 54, 54 * sizeof(double));
  }
}

// Boundary order <-> site-minor order, a tile of 32 sites through shared memory: the boundary side is read or written
// as the contiguous run it is (432 B per site, 576 with CONF's temporal slot), the site-minor side as 512-byte rows.
// EIGEN: the 3x3 blocks of the boundary side are column-major.  Bound by HBM / L2: 14.4 us at 48^3 (6.6 TB/s) against
// 21.8 us with one thread per element and strided 16-byte accesses, 6.5 against 8.0 us at 32^3, 5.1 / 4.9 us at 24^3.
constexpr int kTileSites = 32, kTileThreads = 256;

template <bool TO_SOA>
__global__ void __launch_bounds__(kTileThreads) k_links_tile(double2* __restrict__ bnd, int layout, int V3,
                                                             double2* __restrict__ soa) {
  __shared__ double2 t[27 * kTileSites + 27];  // [site][27], rows of 27: odd, so both sides are conflict-free
  const int s0 = blockIdx.x * kTileSites, ns = min(kTileSites, V3 - s0);
  const int per = layout == LAPH_LAYOUT_CONF ? 36 : 27, skip = per - 27;
  auto element = [&](int e) {  // boundary position of element dir*9 + 3a + b
    if (layout != LAPH_LAYOUT_EIGEN) return e;
    const int d = e / 9, ab = e - d * 9;
    return d * 9 + 3 * (ab % 3) + ab / 3;
  };
  double2* b = bnd + (size_t)s0 * per;
  if (TO_SOA) {
    for (int i = threadIdx.x; i < ns * per; i += kTileThreads) {
      const int s = i / per, e = i - s * per - skip;
      if (e >= 0) t[s * 27 + e] = b[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 27 * kTileSites; i += kTileThreads) {
      const int e = i / kTileSites, s = i - e * kTileSites;
      if (s < ns) soa[(size_t)e * V3 + s0 + s] = t[s * 27 + element(e)];
    }
  } else {
    for (int i = threadIdx.x; i < 27 * kTileSites; i += kTileThreads) {
      const int e = i / kTileSites, s = i - e * kTileSites;
      if (s < ns) t[s * 27 + element(e)] = soa[(size_t)e * V3 + s0 + s];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ns * 27; i += kTileThreads) b[i] = t[i];
  }
}

int links_reorder(double2* bnd, int layout, int V3, double2* soa, bool to_soa, cudaStream_t st) {
  const unsigned nb = ceil_div(V3, kTileSites);
  if (to_soa) k_links_tile<true><<<nb, kTileThreads, 0, st>>>(bnd, layout, V3, soa);
  else k_links_tile<false><<<nb, kTileThreads, 0, st>>>(bnd, layout, V3, soa);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}

int links_to_soa_device(const double* links, int layout, int V3, double2* soa, cudaStream_t st) {
  if (layout != LAPH_LAYOUT_ROWMAJOR && layout != LAPH_LAYOUT_CONF) {
    set_error("links_to_soa_device: layout %d not supported for device links", layout);
    return LAPH_EINVAL;
  }
  LAPH_TRY(links_reorder(reinterpret_cast<double2*>(const_cast<double*>(links)), layout, V3, soa, true, st));
  LAPH_CUDA_TRY(cudaStreamSynchronize(st));
  return LAPH_OK;
}

// The plaquette of every site and plane, p = Re tr(U_d1(s) U_d2(s+d1) U_d1(s+d2)^dag U_d2(s)^dag) / 3, into
// vals[timeslice][plane][site]: one thread each.  The sums below run in one CTA per timeslice, in a fixed order, and
// read 8 bytes per plaquette: 5 + 18 us at 24^3 and 21 + 119 us at 48^3, where one CTA for products and sums took 220 and
// 1690 us.
__global__ void __launch_bounds__(128) k_plaq_vals(const double2* __restrict__ Ub, Lat g, size_t ts_stride,
                                                   double* __restrict__ vals) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x, pl = blockIdx.y;
  if (s >= g.V3) return;
  const double2* U = Ub + blockIdx.z * ts_stride;
  int x, y, z;
  site_xyz(g, s, x, y, z);
  const int d1 = pl == 2 ? 1 : 0, d2 = pl == 0 ? 1 : 2;
  const int j = nb_up(g, x, y, z, d1);
  const int l = nb_up(g, x, y, z, d2);
  const M3 a = m3_mul(ld_link(U, g.V3, s, d1), ld_link(U, g.V3, j, d2));
  const M3 b = m3_mul(ld_link(U, g.V3, s, d2), ld_link(U, g.V3, l, d1));
  // Re tr(a b^dag)
  double tr = 0.0;
#pragma unroll
  for (int e = 0; e < 9; ++e) tr += a.e[e].x * b.e[e].x + a.e[e].y * b.e[e].y;
  vals[((size_t)blockIdx.z * 3 + pl) * g.V3 + s] = tr / 3.0;
}

// Power sums of the plaquettes: one CTA per timeslice, fixed order (deterministic).
__global__ void __launch_bounds__(512) k_plaq_moments(const double* __restrict__ vals, int V3, double* __restrict__ out) {
  const double* v = vals + (size_t)blockIdx.x * 3 * V3;
  double acc[4] = {0, 0, 0, 0};
#pragma unroll 4
  for (int s = threadIdx.x; s < V3; s += 512) {
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) {
      const double p = __ldg(v + (size_t)pl * V3 + s);
      acc[0] += p;
      acc[1] += p * p;
      acc[2] += p * p * p;
      acc[3] += p * p * p * p;
    }
  }
  __shared__ double red[4][512];
#pragma unroll
  for (int k = 0; k < 4; ++k) red[k][threadIdx.x] = acc[k];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
#pragma unroll
      for (int k = 0; k < 4; ++k) red[k][threadIdx.x] += red[k][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 4) out[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

__global__ void k_plaq_finish(const double* __restrict__ mom, int nts, double inv_n, double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nts) out[t] = mom[4 * t] * inv_n;
}

int plaquette_moments_batch(const double2* U, int L, int nts, double* vals, double* out, cudaStream_t st) {
  const Lat g = make_lat(L);
  constexpr int kMaxGridZ = 65535;
  for (int t = 0; t < nts; t += kMaxGridZ)
    k_plaq_vals<<<dim3(ceil_div(g.V3, 128), 3, std::min(kMaxGridZ, nts - t)), 128, 0, st>>>(
        U + (size_t)t * 27 * g.V3, g, (size_t)27 * g.V3, vals + (size_t)t * 3 * g.V3);
  k_plaq_moments<<<nts, 512, 0, st>>>(vals, g.V3, out);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}

int plaquette_batch(const double2* U, int L, int nts, double* vals, double* mom, double* out, cudaStream_t st) {
  LAPH_TRY(plaquette_moments_batch(U, L, nts, vals, mom, st));
  k_plaq_finish<<<ceil_div(nts, 128), 128, 0, st>>>(mom, nts, 1.0 / (3.0 * L * L * L), out);
  LAPH_CUDA_TRY(cudaGetLastError());
  return LAPH_OK;
}

}  // namespace laph
