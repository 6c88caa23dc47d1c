// links.cuh -- link layout conversion at the boundary and per-timeslice
// plaquette reductions (links.cu).
#pragma once
#include "common.cuh"

namespace laph {
// Device links are in site-minor order soa[(dir*9 + 3a + b)*V3 + site] (complex128).
// Host: sites [s0, s0 + n) of the boundary layouts <-> a staging run of 54 doubles per site (the spatial links, in the
// layout's own element order).  links_pack returns the lowest site with a non-finite spatial entry, or -1.
long long links_pack(const double* links, int layout, long long s0, long long n, double* out);
void links_unpack(const double* in, int layout, long long s0, long long n, double* links);
// Device: boundary order (ROWMAJOR, EIGEN, or CONF, whose temporal slot is skipped on the way in and not written on the
// way out) <-> site-minor order.
int links_reorder(double2* bnd, int layout, int V3, double2* soa, bool to_soa, cudaStream_t st);
// Host: LAPH_EINVAL (naming `who` and the first bad site) unless every spatial
// link entry of the host links in `layout` is finite; the temporal slot of
// LAPH_LAYOUT_CONF is not read.  NaN or Inf links would only turn into a solve
// that never converges, so they are refused before any device work.
int check_links_finite(const double* links, int layout, int V3, const char* who);
// Device: same reorder for links already in device memory (ROWMAJOR or CONF).
int links_to_soa_device(const double* links, int layout, int V3, double2* soa, cudaStream_t st);
// Device: average spatial plaquette of nts timeslices -> out[nts]
// (plaque_timeslice, modules/config_utils.cpp:388-426).  Scratch: vals[3 V3 nts], mom[4 nts].
int plaquette_batch(const double2* U, int L, int nts, double* vals, double* mom, double* out, cudaStream_t st);
// Device: power sums of the per-(site, plane) plaquette p = Re tr P / 3:
// out[ts*4 + k] = sum p^(k+1) over 3*V3 values, k = 0..3.  Scratch: vals[3 V3 nts].
int plaquette_moments_batch(const double2* U, int L, int nts, double* vals, double* out, cudaStream_t st);
}  // namespace laph
