// PCG of a small C3D10 system in one kernel (small_solve.cu).
#pragma once

#include <cuda_runtime.h>

#include "amg.h"
#include "solid.h"

namespace wn {

// Solves K x = b from x = 0 to ||r|| <= rtol ||b|| (x in W.p64.x) with the preconditioner in TM and
// copies the result's scalars to hS.  0: done; 1: for the launched kernels (not a small system, or no
// room for the cluster); anything else: an error.
template <typename TM>
int small_pcg(Solid* s, SolverWork& W, const double* b, double rtol, int max_iter, int precond, PcgScalars* S,
              cudaStream_t st, PcgScalars* hS);

}  // namespace wn
