// Declarations shared by the FNO's general kernels (fno.cu) and its fused ones (fno_fused.cu).
#pragma once
#include <cuda_runtime.h>

namespace pg {

// Address of the flag that a kernel sets when a bounded wait gave up (pg_gemm_timeouts reads it).
cudaError_t gemm_timeout_flag(int** flag);
// 0: tcgen05, 1: mma.sync (pg_gemm_set_engine).
int gemm_engine();
// Polls of a fused kernel's completion waits, 0 for the give-up setting (pg_gemm_set_wait_limit).  The bound
// itself is compiled in: read from the arguments it made a training pass 2 % slower.
int gemm_wait_limit();

// Shared memory of a block at most.
constexpr int kMaxSmem = 227 * 1024;

// Allows `kernel` all of it but `fixed` bytes of static shared memory.  The limit belongs to the
// kernel on a device, not to a launch: every caller asks for the same one, whatever its launch takes,
// so that one thread's small launch never lowers the limit under another's large one.
template <typename K>
cudaError_t allow_smem(K* kernel, int fixed = 0) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - fixed);
}

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
