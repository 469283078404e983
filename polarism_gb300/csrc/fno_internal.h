// Declarations shared by the FNO's general kernels (fno.cu) and its fused ones (fno_fused.cu).
#pragma once
#include <cuda_runtime.h>

namespace pg {

// Address of the flag that a kernel sets when a bounded wait gave up (pg_gemm_timeouts reads it).
cudaError_t gemm_timeout_flag(int** flag);
// 0: tcgen05, 1: mma.sync (pg_gemm_set_engine).
int gemm_engine();

// GELU in its tanh form and its derivative.
constexpr float kGeluC = 0.7978845608028654f;  // sqrt(2 / pi)

__device__ __forceinline__ float gelu_f(float x) {
  return 0.5f * x * (1.f + tanhf(kGeluC * (x + 0.044715f * x * x * x)));
}

__device__ __forceinline__ float gelu_grad_f(float x) {
  const float t = tanhf(kGeluC * (x + 0.044715f * x * x * x));
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * kGeluC * (1.f + 3.f * 0.044715f * x * x);
}

}  // namespace pg
