// Split-step passes on the register-resident transforms (fft_reg.cuh): rows and columns of 64 to
// 4096 points.  The passes, their order and the local operations are those of split.cu.
//
// Row pass: a row's values come straight from global memory into registers (lane-consecutive),
// are transformed, kicked, transformed back and stored.  Column pass: a panel of columns, the
// inverse transform, the local step on each thread's own sixteen sites -- kept in the thread's
// own slots of the exchange buffer, so that the step is one loop over batches of sites whose
// reservoir and envelope loads are all issued before the first site's arithmetic -- and the
// forward transform.  An inverse transform is the forward one of the conjugate, conjugated.
#pragma once
#include "reg_pass.cuh"
#include "split_local.cuh"

namespace pg {
namespace {

template <typename T, int N, int V>
__global__ void __launch_bounds__(RowShape<N, V, 1>::MAX_THREADS, sizeof(T) == 4 ? 1024 / RowShape<N, V, 1>::MAX_THREADS
                                                                              : 512 / RowShape<N, V, 1>::MAX_THREADS)
    row_reg_kernel(typename C2T<T>::type* __restrict__ data,
                   const typename TwEntry<T>::type* __restrict__ tab,
                   const typename C2T<T>::type* __restrict__ px,
                   const typename C2T<T>::type* __restrict__ py, const RowPassArgs a) {
  using C2 = typename C2T<T>::type;
  using S = RowShape<N, V, 1>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.halt != nullptr && __ldcg(a.halt) != 0) return;  // steady-state monitor halted the run
  const int t = threadIdx.x % S::M, r = threadIdx.x / S::M;
  const int member = blockIdx.z;
  const int row = blockIdx.x * a.rows + r;
  C2* buf = reinterpret_cast<C2*>(smem_raw) + r * S::STRIDE;
  const GroupSync<(S::M <= 32)> sync{1 + r, S::M};
  C2* d = data + (static_cast<long long>(member) * a.ny + row) * N + t;
  C2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = d[m * S::M];
  // Phase 0: forward transform and kick; phase 1: the inverse transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.forward : a.inverse) {
      if (ph == 1) conj_all(v);
      fft_forward<T, N, V>(v, t, buf, 1, tab, sync);
      if (ph == 1) conj_all(v);
    }
    if (ph == 0 && a.multiply) {
      const C2* pxm = px + static_cast<long long>(member) * a.table_stride + t;
      const C2 dy = py[static_cast<long long>(member) * a.table_stride + row];
      const T scale = static_cast<T>(a.scale);
#pragma unroll
      for (int m = 0; m < V; ++m) v[m] = kick(v[m], pxm[m * S::M], dy, scale);
    }
  }
#pragma unroll
  for (int m = 0; m < V; ++m) d[m * S::M] = v[m];
}

// The local step on a thread's own sites, BATCH at a time with the batch's loads first; SINGLE:
// the single case (LocalStep::single).
template <typename T, int N, int V, int BATCH, bool SINGLE, int OP, bool NOISE>
__device__ __forceinline__ void own_local(const LocalStep<T>& local, typename C2T<T>::type* buf, int C,
                                          int t, int nx, int x) {
  using C2 = typename C2T<T>::type;
  const OwnSlots<N, V> own(t);
#pragma unroll 1
  for (int m0 = 0; m0 < V; m0 += BATCH) {
    int o[BATCH];
    typename LocalStep<T>::Inputs in[BATCH];
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
      C2 v = buf[own.slot(m0 + u) * C];
      if (SINGLE)
        in[u].n = local.template step_single<OP, NOISE>(v, in[u].n, in[u].Pa, o[u]);
      else
        local.template compute<OP, NOISE>(v, in[u], o[u]);
      buf[own.slot(m0 + u) * C] = v;
      if (SINGLE) {
        if (OP != SPLIT_OP_NONLINEAR) local.rm[o[u]] = in[u].n;
      } else {
        local.store(in[u], o[u]);
      }
    }
  }
}

template <typename T, int N, int V, int BATCH, bool SINGLE>
__device__ __forceinline__ void own_local_run(const LocalStep<T>& local, typename C2T<T>::type* buf, int C,
                                              int t, int nx, int x) {
  switch (local.op * 2 + (local.noise ? 1 : 0)) {
#define PG_SPLIT_OWN(OP, NOISE)                                            \
  case OP * 2 + NOISE:                                                     \
    own_local<T, N, V, BATCH, SINGLE, OP, NOISE>(local, buf, C, t, nx, x);    \
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

template <typename T, int N, int V>
__global__ void __launch_bounds__(ColShape<T, N, V, 1>::MAX_THREADS, ColShape<T, N, V, 1>::MIN_BLOCKS)
    col_reg_kernel(typename C2T<T>::type* __restrict__ data, T* __restrict__ res,
                   const T* __restrict__ pump, const T* __restrict__ potential,
                   const typename TwEntry<T>::type* __restrict__ tab,
                   const SplitConst<T>* __restrict__ consts, const T* __restrict__ scales,
                   const unsigned long long* __restrict__ step_base, const ColPassArgs a) {
  using C2 = typename C2T<T>::type;
  constexpr int M = RegFft<N, V>::M;
  constexpr int kBatch = 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.halt != nullptr && __ldcg(a.halt) != 0) return;  // steady-state monitor halted the run
  const int C = a.cols;
  const int c = threadIdx.x & (C - 1), t = threadIdx.x >> a.log2cols;
  const int member = blockIdx.z;
  const int x = blockIdx.x * C + c;
  const int nx = a.nx;
  C2* buf = reinterpret_cast<C2*>(smem_raw) + c;
  C2* d = data + static_cast<long long>(member) * nx * N + x;
  C2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = d[static_cast<long long>(t + M * m) * nx];
  // Phase 0: the inverse transform and the local step; phase 1: the forward transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.inverse : a.forward) {
      if (ph == 0) conj_all(v);
      fft_forward<T, N, V>(v, t, buf, C, tab, BlockSync{});
      if (ph == 0) conj_all(v);
    }
    if (ph == 1 || a.op == SPLIT_OP_NONE) continue;
    const OwnSlots<N, V> own(t);
#pragma unroll
    for (int m = 0; m < V; ++m) buf[own.slot(m) * C] = v[m];
    const LocalStep<T> local(a, member, res, pump, potential, consts, scales, step_base);
    if (local.single())
      own_local_run<T, N, V, kBatch, true>(local, buf, C, t, nx, x);
    else
      own_local_run<T, N, V, kBatch, false>(local, buf, C, t, nx, x);
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = buf[own.slot(m) * C];
  }
#pragma unroll
  for (int m = 0; m < V; ++m) d[static_cast<long long>(t + M * m) * nx] = v[m];
}

template <typename T>
cudaError_t configure_row_reg(int nx) {
#define PG_X(N, V)                                                                                     \
  return cudaFuncSetAttribute(row_reg_kernel<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                              static_cast<int>(RowShape<N, V, 1>::MAX_THREADS / RowShape<N, V, 1>::M * \
                                               RowShape<N, V, 1>::STRIDE * 2 * sizeof(T)))
  PG_REG_SIZES(nx, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

template <typename T>
cudaError_t configure_col_reg(int ny) {
#define PG_X(N, V)                                                                                  \
  return cudaFuncSetAttribute(col_reg_kernel<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                              static_cast<int>(ColShape<T, N, V, 1>::MAX_COLS *                     \
                                               ColShape<T, N, V, 1>::SLOTS * 2 * sizeof(T)))
  PG_REG_SIZES(ny, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

template <typename T>
cudaError_t launch_row_reg_t(T* data, const T* tab, const T* px, const T* py, RowPassArgs a, int members, int sm_count, cudaStream_t stream) {
  using C2 = typename C2T<T>::type;
#define PG_X(N, V)                                                                                 \
  {                                                                                                \
    using S = RowShape<N, V, 1>;                                                                   \
    a.rows = row_shape_rows<N, V, 1>(a.ny, members, sm_count);                                     \
    row_reg_kernel<T, N, V><<<dim3(a.ny / a.rows, 1, members), a.rows * S::M,                      \
                              static_cast<size_t>(a.rows) * S::STRIDE * sizeof(C2), stream>>>(     \
        reinterpret_cast<C2*>(data), reinterpret_cast<const typename TwEntry<T>::type*>(tab),      \
        reinterpret_cast<const C2*>(px), reinterpret_cast<const C2*>(py), a);                      \
    return cudaGetLastError();                                                                     \
  }
  PG_REG_SIZES(a.nx, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

template <typename T>
cudaError_t launch_col_reg_t(T* data, T* res, const T* pump, const T* potential, const T* tab,
                             const SplitConst<T>* consts, const T* scales,
                             const unsigned long long* step_base, ColPassArgs a, int sm_count,
                             cudaStream_t stream) {
  using C2 = typename C2T<T>::type;
#define PG_X(N, V)                                                                                    \
  {                                                                                                   \
    a.cols = col_shape_cols<T, N, V, 1>(a.nx, a.members, sm_count);                                   \
    a.log2cols = log2_of(a.cols);                                                                     \
    col_reg_kernel<T, N, V><<<dim3(a.nx / a.cols, 1, a.members), a.cols * RegFft<N, V>::M,            \
                              static_cast<size_t>(a.cols) * RegFft<N, V>::SLOTS * sizeof(C2), stream>>>( \
        reinterpret_cast<C2*>(data), res, pump, potential,                                            \
        reinterpret_cast<const typename TwEntry<T>::type*>(tab), consts, scales, step_base, a);       \
    return cudaGetLastError();                                                                        \
  }
  PG_REG_SIZES(a.ny, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

}  // namespace
}  // namespace pg
