// FP32 split-step passes on the register-resident transforms (fft_reg.cuh): rows and columns of 64 to
// 4096 points.  The passes, their order and the local operations are those of split.cu.
//
// Row pass: a row's values come straight from global memory into registers (lane-consecutive),
// are transformed, kicked, transformed back and stored.  Column pass: a panel of columns, the
// inverse transform, the local step on each thread's own sites -- kept in the thread's
// own slots of the exchange buffer, so that the step is one loop over batches of sites whose
// reservoir and envelope loads are all issued before the first site's arithmetic -- and the
// forward transform.  An inverse transform is the forward one of the conjugate, conjugated.
#include "reg_pass.cuh"
#include "split_local.cuh"

namespace pg {
namespace {

template <int N, int V>
__global__ void __launch_bounds__(RowShape<N, V, 1>::MAX_THREADS, 1024 / RowShape<N, V, 1>::MAX_THREADS)
    row_reg_kernel(float2* __restrict__ data, const float4* __restrict__ tab, const float2* __restrict__ px,
                   const float2* __restrict__ py, const RowPassArgs a) {
  using S = RowShape<N, V, 1>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.halt != nullptr && __ldcg(a.halt) != 0) return;  // steady-state monitor halted the run
  const int t = threadIdx.x % S::M, r = threadIdx.x / S::M;
  const int member = blockIdx.z;
  const int row = blockIdx.x * a.rows + r;
  float2* buf = reinterpret_cast<float2*>(smem_raw) + r * S::STRIDE;
  const GroupSync<(S::M <= 32)> sync{1 + r, S::M};
  float2* d = data + (static_cast<long long>(member) * a.ny + row) * N + t;
  float2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = d[m * S::M];
  // Phase 0: forward transform and kick; phase 1: the inverse transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.forward : a.inverse) {
      if (ph == 1) conj_all(v);
      fft_forward<N, V>(v, t, buf, 1, tab, sync);
      if (ph == 1) conj_all(v);
    }
    if (ph == 0 && a.multiply) {
      const float2* pxm = px + static_cast<long long>(member) * a.table_stride + t;
      const float2 dy = py[static_cast<long long>(member) * a.table_stride + row];
      const float scale = static_cast<float>(a.scale);
#pragma unroll
      for (int m = 0; m < V; ++m) v[m] = kick(v[m], pxm[m * S::M], dy, scale);
    }
  }
#pragma unroll
  for (int m = 0; m < V; ++m) d[m * S::M] = v[m];
}

// The local step on a thread's own sites, BATCH at a time with the batch's loads first; SINGLE:
// the single case (LocalStep::single).
template <int N, int V, int BATCH, bool SINGLE, int OP, bool NOISE>
__device__ __forceinline__ void own_local(const LocalStep<float>& local, float2* buf, int C, int t, int nx, int x) {
  const OwnSlots<N, V> own(t);
#pragma unroll 1
  for (int m0 = 0; m0 < V; m0 += BATCH) {
    int o[BATCH];
    LocalStep<float>::Inputs in[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      o[u] = (t + RegFft<N, V>::M * (m0 + u)) * nx + x;
      if (SINGLE) {
        in[u].n = local.rm[o[u]];
        in[u].Pa = local.pm[o[u]];
      } else {
        in[u] = local.load(o[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      float2 v = buf[own.slot(m0 + u) * C];
      if (SINGLE)
        in[u].n = local.step_single<OP, NOISE>(v, in[u].n, in[u].Pa, o[u]);
      else
        local.compute<OP, NOISE>(v, in[u], o[u]);
      buf[own.slot(m0 + u) * C] = v;
      if (SINGLE) {
        if (OP != SPLIT_OP_NONLINEAR) local.rm[o[u]] = in[u].n;
      } else {
        local.store(in[u], o[u]);
      }
    }
  }
}

template <int N, int V, int BATCH, bool SINGLE>
__device__ __forceinline__ void own_local_run(const LocalStep<float>& local, float2* buf, int C, int t, int nx, int x) {
  switch (local.op * 2 + (local.noise ? 1 : 0)) {
#define PG_SPLIT_OWN(OP, NOISE)                                            \
  case OP * 2 + NOISE:                                                     \
    own_local<N, V, BATCH, SINGLE, OP, NOISE>(local, buf, C, t, nx, x);       \
    break;
    PG_SPLIT_OWN(SPLIT_OP_KOUTER, 1)
    PG_SPLIT_OWN(SPLIT_OP_KOUTER, 0)
    PG_SPLIT_OWN(SPLIT_OP_NONLINEAR, 1)
    PG_SPLIT_OWN(SPLIT_OP_NONLINEAR, 0)
    case SPLIT_OP_RES_START * 2 + 1:
    PG_SPLIT_OWN(SPLIT_OP_RES_START, 0)
    case SPLIT_OP_RES_END * 2 + 1:
    PG_SPLIT_OWN(SPLIT_OP_RES_END, 0)
    case SPLIT_OP_RES_END_START * 2 + 1:
    PG_SPLIT_OWN(SPLIT_OP_RES_END_START, 0)
#undef PG_SPLIT_OWN
    default:
      break;
  }
}

template <int N, int V>
__global__ void __launch_bounds__(ColShape<N, V, 1>::MAX_THREADS, ColShape<N, V, 1>::MIN_BLOCKS)
    col_reg_kernel(float2* __restrict__ data, float* __restrict__ res, const float* __restrict__ pump,
                   const float* __restrict__ potential, const float4* __restrict__ tab,
                   const SplitConst<float>* __restrict__ consts, const float* __restrict__ scales,
                   const unsigned long long* __restrict__ step_base, const ColPassArgs a) {
  constexpr int M = RegFft<N, V>::M;
  constexpr int kBatch = 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.halt != nullptr && __ldcg(a.halt) != 0) return;  // steady-state monitor halted the run
  const int C = a.cols;
  const int c = threadIdx.x & (C - 1), t = threadIdx.x >> a.log2cols;
  const int member = blockIdx.z;
  const int x = blockIdx.x * C + c;
  const int nx = a.nx;
  float2* buf = reinterpret_cast<float2*>(smem_raw) + c;
  float2* d = data + static_cast<long long>(member) * nx * N + x;
  float2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = d[static_cast<long long>(t + M * m) * nx];
  // Phase 0: the inverse transform and the local step; phase 1: the forward transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.inverse : a.forward) {
      if (ph == 0) conj_all(v);
      fft_forward<N, V>(v, t, buf, C, tab, BlockSync{});
      if (ph == 0) conj_all(v);
    }
    if (ph == 1 || a.op == SPLIT_OP_NONE) continue;
    const OwnSlots<N, V> own(t);
#pragma unroll
    for (int m = 0; m < V; ++m) buf[own.slot(m) * C] = v[m];
    const LocalStep<float> local(a, member, res, pump, potential, consts, scales, step_base);
    if (local.single())
      own_local_run<N, V, kBatch, true>(local, buf, C, t, nx, x);
    else
      own_local_run<N, V, kBatch, false>(local, buf, C, t, nx, x);
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = buf[own.slot(m) * C];
  }
#pragma unroll
  for (int m = 0; m < V; ++m) d[static_cast<long long>(t + M * m) * nx] = v[m];
}

cudaError_t configure_row_reg(int nx) {
#define PG_X(N, V)                                                                                   \
  return cudaFuncSetAttribute(row_reg_kernel<N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                              static_cast<int>(RowShape<N, V, 1>::MAX_THREADS / RowShape<N, V, 1>::M * \
                                               RowShape<N, V, 1>::STRIDE * sizeof(float2)))
  PG_REG_SIZES(nx, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

cudaError_t configure_col_reg(int ny) {
#define PG_X(N, V)                                                                                \
  return cudaFuncSetAttribute(col_reg_kernel<N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                              static_cast<int>(ColShape<N, V, 1>::MAX_COLS * ColShape<N, V, 1>::SLOTS * sizeof(float2)))
  PG_REG_SIZES(ny, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

}  // namespace

cudaError_t configure_split_reg(int nx, int ny) {
  if (reg_fft_size(nx)) {
    const cudaError_t e = configure_row_reg(nx);
    if (e != cudaSuccess) return e;
  }
  return reg_fft_size(ny) ? configure_col_reg(ny) : cudaSuccess;
}

cudaError_t launch_row_reg(float* data, const float* tab, const float* px, const float* py,
                           const RowPassArgs& args, int members, int sm_count, cudaStream_t stream) {
  RowPassArgs a = args;
#define PG_X(N, V)                                                                                 \
  {                                                                                                \
    using S = RowShape<N, V, 1>;                                                                   \
    a.rows = row_shape_rows<N, V, 1>(a.ny, members, sm_count);                                     \
    row_reg_kernel<N, V><<<dim3(a.ny / a.rows, 1, members), a.rows * S::M,                         \
                           static_cast<size_t>(a.rows) * S::STRIDE * sizeof(float2), stream>>>(    \
        reinterpret_cast<float2*>(data), reinterpret_cast<const float4*>(tab),                     \
        reinterpret_cast<const float2*>(px), reinterpret_cast<const float2*>(py), a);              \
    return cudaGetLastError();                                                                     \
  }
  PG_REG_SIZES(a.nx, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

cudaError_t launch_col_reg(float* data, float* res, const float* pump, const float* potential,
                           const float* tab, const SplitConst<float>* consts, const float* scales,
                           const unsigned long long* step_base, const ColPassArgs& args, int sm_count,
                           cudaStream_t stream) {
  ColPassArgs a = args;
#define PG_X(N, V)                                                                                    \
  {                                                                                                   \
    a.cols = col_shape_cols<N, V, 1>(a.nx, a.members, sm_count);                                      \
    a.log2cols = log2_of(a.cols);                                                                     \
    col_reg_kernel<N, V><<<dim3(a.nx / a.cols, 1, a.members), a.cols * RegFft<N, V>::M,               \
                           static_cast<size_t>(a.cols) * RegFft<N, V>::SLOTS * sizeof(float2), stream>>>( \
        reinterpret_cast<float2*>(data), res, pump, potential, reinterpret_cast<const float4*>(tab),  \
        consts, scales, step_base, a);                                                                \
    return cudaGetLastError();                                                                        \
  }
  PG_REG_SIZES(a.ny, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

}  // namespace pg
