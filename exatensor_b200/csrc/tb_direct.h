// tb_direct.h -- one-kernel contractions in the tensors' own layouts (tb_direct.cu).
#pragma once
#include <cuda_runtime.h>

#include "tb_direct_plan.h"

namespace tb {

// plan_direct over the kernels' tile shapes on the current device.
int direct_plan(const Matricization& Z, int dtk, const void* d, const void* l, const void* r, DirectPlan* out);
// Launches it; alpha as the plain method takes it (real kinds: ai = 0).  `when` (R8, C8): a
// device word; the kernel does nothing unless it is set.
int run_direct(const DirectPlan& plan, int dtk, double ar, double ai, bool accumulate, int lconj, int rconj,
               cudaStream_t s, const unsigned* when = nullptr);

}  // namespace tb
