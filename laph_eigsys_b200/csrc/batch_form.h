// batch_form.h -- the kernels a solver picks by the size of its whole batch.
// The autotuner times solves of a sample of a batch, which has to run the
// kernels of the batch, not those a batch as small as the sample would take:
// it creates its solvers with laph_solver_create_for.  Exported, but not part of
// the public interface.
#pragma once
#include "../../include/laph_gpu.h"

namespace laph {
struct BatchForm {
  int pass;        // the filter runs each whole pass as one kernel per extent
  int block;       // columns per CTA of the filter's step kernels
  int cols64;      // columns per CTA of the FP64 block stencils
  int gram_split;  // the Gram takes its kernel for few units
  int kmax;        // widest block
};
// The form of a batch with these options on `device` (problems and options already checked).
int batch_form(const laph_problem* batch, int n, const laph_solve_opts* opts, int device, BatchForm* f);
}  // namespace laph

extern "C" {
// laph_solver_create for probs[0..n), with the kernels of batch[0..nbatch), of which they are a sample.
int laph_solver_create_for(laph_solver** out, const laph_problem* probs, int n, const laph_solve_opts* opts, int device,
                           const laph_problem* batch, int nbatch);
// Columns per CTA of the solver's filter, and whether its passes run as one kernel each.
int laph_solver_form(laph_solver* s, int* block, int* pass);
// Blocks wider than `width` run their Jacobi in global memory, as they do on a device without room for their clusters
// (for the tests; before the solver's first run).
int laph_solver_limit_jacobi(laph_solver* s, int width);
}
