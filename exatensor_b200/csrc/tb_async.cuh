// tb_async.cuh -- device instructions shared by the kernels that stage operands
// element by element and multiply in FP64.
#pragma once
#include <cstdint>

namespace tb {

// Asynchronous copy of one element into shared memory; zero-filled when !valid (src is
// then any valid address and is not read).
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* sdst, const void* gsrc, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(sdst);
  const int n = valid ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(gsrc), "n"(BYTES), "r"(n) : "memory");
}

// 8 x 8 x 4 FP64 tensor-core product: one element of A and of B and two sums per lane.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

}  // namespace tb
