// Launch shapes and synchronisation shared by the register-resident row and column passes
// (split_reg.cu, ifrk_reg.cu).
#pragma once
#include <algorithm>

#include "fft_reg.cuh"

namespace pg {
namespace {

// The element `bytes` past a block-uniform base.
template <typename E>
__device__ __forceinline__ const E& at_offset(const E* base, unsigned bytes) {
  return *reinterpret_cast<const E*>(reinterpret_cast<const char*>(base) + bytes);
}
template <typename E>
__device__ __forceinline__ E& at_offset(E* base, unsigned bytes) {
  return *reinterpret_cast<E*>(reinterpret_cast<char*>(base) + bytes);
}

// Barrier over the threads of one transform (or of a row's transforms): within a warp, or a named
// barrier of `count` threads.
template <bool WARP>
struct GroupSync {
  int id, count;
  __device__ __forceinline__ void operator()() const {
    if constexpr (WARP)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
  }
};
struct BlockSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// Row pass: `rows` rows of COMPS components a block, N / V threads each.  Rows of fewer than 16
// threads share half-warps: their buffers are offset so that the half-warp's accesses stay on
// distinct banks.
template <int N, int V, int COMPS>
struct RowShape {
  static constexpr int M = RegFft<N, V>::M;
  static constexpr int GROUP = M * COMPS;  // threads of one row
  static constexpr int STRIDE = RegFft<N, V>::SLOTS + (M < 16 ? M : 0);
  static constexpr int MAX_THREADS = GROUP > 256 ? GROUP : 256;
};

// Rows a block: 256 threads, fewer (down to a warp, or one row) where the grid would not give two
// blocks an SM.
template <int N, int V, int COMPS>
int row_shape_rows(int ny, int members, int sm_count) {
  using S = RowShape<N, V, COMPS>;
  int rows = std::max(1, std::min(ny, 256 / S::GROUP));
  while (rows > 1 && rows / 2 * S::GROUP >= 32 &&
         static_cast<long long>(ny / rows) * members < 2LL * sm_count)
    rows /= 2;
  return rows;
}

// Column pass: `cols` columns of COMPS components a block.
template <int N, int V, int COMPS>
struct ColShape {
  static constexpr int M = RegFft<N, V>::M;
  static constexpr int SLOTS = RegFft<N, V>::SLOTS;
  static constexpr int REGS = 64;  // a thread
  // 64-byte row segments (8 columns) while the block stays within 1024 threads.
  static constexpr int cap(int want) {
    int c = want;
    while (c > 1 && c * M * COMPS > 1024) c /= 2;
    return c;
  }
  static constexpr int MAX_COLS = cap(8);
  static constexpr int MAX_THREADS = MAX_COLS * M * COMPS < 32 ? 32 : MAX_COLS * M * COMPS;
  static constexpr int MIN_BLOCKS = 65536 / (REGS * (MAX_THREADS < 128 ? 128 : MAX_THREADS));
};

template <int N, int V, int COMPS>
int col_shape_cols(int nx, int members, int sm_count) {
  using S = ColShape<N, V, COMPS>;
  int cols = std::min(S::MAX_COLS, nx);
  while (cols > 2 && cols / 2 * S::M * COMPS >= 32 &&
         5LL * (nx / cols) * members < 4LL * sm_count)
    cols /= 2;
  return cols;
}

// A switch over the sizes of the passes: X(N, V) for n points (V as reg_fft_vals).
#define PG_REG_SIZES(n, X) \
  switch (n) {             \
    case 64: X(64, 8);     \
    case 128: X(128, 8);   \
    case 256: X(256, 8);   \
    case 512: X(512, 8);   \
    case 1024: X(1024, 16); \
    case 2048: X(2048, 16); \
    case 4096: X(4096, 16); \
    default: break;        \
  }

inline int log2_of(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

}  // namespace
}  // namespace pg
