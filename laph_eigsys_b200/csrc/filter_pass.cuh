// filter_pass.cuh -- a whole Chebyshev pass of the filter as one kernel per
// lattice extent (filter_pass.cu).
#pragma once
#include <vector>

#include "batch.cuh"

namespace laph {

// The problems of one extent L and how a pass over them is laid out: `teams`
// teams of `tiles` CTAs, ns sites each, every team filtering `gmax` columns of
// one problem at a time at most.
struct PassClass {
  int L, ns, tiles, teams, gmax;
};

// Layout of a pass for these problems on the current device; empty where the
// step kernels are the faster ones (batches of many site-columns) or the only
// ones (an extent whose sites outnumber the co-resident threads, or more than
// kPassClasses extents).
constexpr int kPassClasses = 4;
// Have the problems few enough site-columns and extents for it?  Fed one by one.
struct PassSize {
  long long work = 0;
  int extents = 0, seen[kPassClasses] = {};
  void add(int L, int k);
  bool small() const;
};
int pass_layout(const std::vector<ProbDesc>& probs, int bf16, std::vector<PassClass>* out);
// ints of plan scratch for np problems
size_t pass_plan_ints(int np);
// All steps n = 1 .. m-1 of a pass (m = *dm when dm is not null) on every unlocked
// column of every active problem, W = V on the locked ones; E0, E1: scratch of
// the size of a vector block; plan: pass_plan_ints(np) ints; *err is set (and
// the pass left unfinished) when a wait between CTAs gives up.
int filter_pass(const std::vector<PassClass>& cls, const ProbDesc* pd, const ProbState* ps, int np, int bf16,
                const void* links, const float* scale, const float2* S, float2* E0, float2* E1, const double2* V,
                double2* W, const double* tcoef, int m, const int* dm, int* plan, int* err, cudaStream_t st);
// kernels one filter_pass launches
inline int pass_launches(const std::vector<PassClass>& cls) { return 1 + (int)cls.size(); }

}  // namespace laph
