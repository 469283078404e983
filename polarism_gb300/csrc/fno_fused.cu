// Fused kernels of the Fourier neural operator on tcgen05: one launch per pass over the activations.
//
// The maps are those of fno.cu's general GEMM with the same BF16 operands, the same 16-wide K steps in
// ascending order and the same FP32 operations after them, so the results are its results; what is
// left out is memory traffic and latency.  The activations of a layer are [sample][channel][y][x] with a
// few dozen channels: a GEMM with the channels as M filled a quarter of a 128-row tile and wrote its
// FP32 product for a second GEMM to read, add and write, and for elementwise passes after it.  Here the
// pixels are the 128 rows of a tile and the channels its columns: x is contiguous, so operands are copied as
// they lie (16 bytes a copy, M-major), a warp's 32 lanes hold 32 consecutive x of one channel for the
// epilogue, and the epilogue finishes the layer (spectral term, bias, GELU or its derivative, BF16).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fno_internal.h"
#include "pg_internal.h"
#include "tc05.cuh"
#include "tma.cuh"

namespace pg {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kThreads = 128;
// Layouts: the strides between core matrices carry 16 spare bytes where neighbouring lanes of a copy
// would otherwise write the same banks.
constexpr int kMnChunk = 144;              // M-major operand of 128 rows: 8 rows of M to the next 8
constexpr int kMnGroup = 16 * kMnChunk;    // and 8 k to the next 8
__host__ __device__ constexpr int pad16(int v) { return (v + 15) & ~15; }
__host__ __device__ constexpr int pad8(int v) { return (v + 7) & ~7; }
// K-major operand of `rows` rows (a multiple of 8): 8 k to the next 8; row groups are 128 bytes apart.
__host__ __device__ constexpr int k_group(int rows) { return rows * 16 + 16; }

__device__ __forceinline__ void zero_smem(unsigned char* p, int bytes) {
  for (int o = threadIdx.x * 16; o < bytes; o += kThreads * 16)
    *reinterpret_cast<uint4*>(p + o) = make_uint4(0u, 0u, 0u, 0u);
}

// The block's copies of an operand, `groups` 16-byte groups a row, into its core matrices.  Lanes run along a
// row, `WIDTH` of them (a power of two), so that no index is divided; 16 spare bytes between groups
// keep their writes on different banks.
// K-major: group j of row r at dst + j * group + 16 r.
template <int WIDTH>
__device__ __forceinline__ void copy_k_major_w(unsigned char* dst, int group, const bf16* src, long long ld, int rows,
                                               int groups) {
  const int j0 = threadIdx.x % WIDTH;
  for (int j = j0; j < groups; j += WIDTH) {
    const int r0 = threadIdx.x / WIDTH;
    const bf16* p = src + r0 * ld + j * 8;
    unsigned char* d = dst + j * group + r0 * 16;
#pragma unroll 4
    for (int r = r0; r < rows; r += kThreads / WIDTH, p += kThreads / WIDTH * ld, d += kThreads / WIDTH * 16)
      cp_async16(d, p);
  }
}
__device__ __forceinline__ void copy_k_major(unsigned char* dst, int group, const bf16* src, long long ld, int rows,
                                             int groups) {
  if (groups <= 4)
    copy_k_major_w<4>(dst, group, src, ld, rows, groups);
  else if (groups <= 8)
    copy_k_major_w<8>(dst, group, src, ld, rows, groups);
  else
    copy_k_major_w<32>(dst, group, src, ld, rows, groups);
}
// M- or N-major: group c of row k at dst + (k / 8) group + c kMnChunk + (k % 8) 16.
template <int WIDTH>
__device__ __forceinline__ void copy_mn_major_w(unsigned char* dst, int group, const bf16* src, long long ld, int rows,
                                                int groups) {
  const int c = threadIdx.x % WIDTH;
  if (c >= groups) return;
  const int k0 = threadIdx.x / WIDTH;
  const bf16* p = src + k0 * ld + c * 8;
#pragma unroll 4
  for (int k = k0; k < rows; k += kThreads / WIDTH, p += kThreads / WIDTH * ld)
    cp_async16(dst + (k >> 3) * group + c * kMnChunk + (k & 7) * 16, p);
}
__device__ __forceinline__ void copy_mn_major(unsigned char* dst, int group, const bf16* src, long long ld, int rows,
                                              int groups) {  // at most 16 groups
  if (groups <= 4)
    copy_mn_major_w<4>(dst, group, src, ld, rows, groups);
  else
    copy_mn_major_w<16>(dst, group, src, ld, rows, groups);
}

// One TMEM allocation and one completion barrier per block; `cols` columns.
__device__ __forceinline__ uint32_t tc_begin(uint64_t* mbar, int barriers, uint32_t* slot, uint32_t cols) {
  if (threadIdx.x < 32) tc_alloc(smem_u32(slot), cols);
  if (threadIdx.x == 0) {
    for (int q = 0; q < barriers; ++q) mbar_init(smem_u32(mbar + q), 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *slot;
}
// `drain` is a barrier that nothing else uses.  A thread whose wait gave up does not leave the loops
// (the block's barriers stay matched): it stops waiting and storing; the issuing thread waits here, bounded,
// for whatever products are still in flight before the accumulators are freed.
__device__ __forceinline__ void tc_end(uint32_t tmem, uint32_t cols, bool ok, uint64_t* drain, int* err_flag) {
  if (!ok) {
    atomicOr(err_flag, 1);
    if (threadIdx.x == 0) {
      tc_commit(smem_u32(drain));
      mbar_wait_bounded(smem_u32(drain), 0u, kTcWaitLimit);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tc_dealloc(tmem, cols);
}

// ---------------------------------------------------------------------------------- layer
constexpr int kLayerBlocks = 6;  // blocks an SM, where shared and tensor memory allow them

struct LayerArgs {
  const bf16* w;      // [cout][cin], or [cin][cout] when w_t
  const bf16* v;      // [B][cin][n][n]
  const bf16* z;      // spectral term: [B][cout][n][k2], or null
  const bf16* table;  // [k2][n], or [n][k2] when table_rows
  const float* bias;  // [cout] or null
  const float* pre;   // mode 2: [B][cout][n][n]
  float* u;           // [B][cout][n][n] or null
  bf16* out;          // [B][cout][n][n] or null
  int w_t, table_rows, cin, cout, n, B, k2;
  int o_t, o_v, o_z, o_bar, cols;  // shared-memory offsets (w at 0) and TMEM columns
  int v_bytes, z_bytes;            // of one of the two buffers
  int waits;                       // 0: the give-up setting, every completion wait has failed
};

// x[b, co, p] = sum_k w[co, k] v[b, k, p] + sum_q z[b, co, y, q] table[q, x] + bias[co] for the pixels
// p = (y, x) of one tile of at most 128 x in a row; persistent over the rows.  MODE 0: u = out = x;
// 1: u = x, out = gelu(x); 2: u = out = x gelu'(pre).  The
// next row's v and z are in flight while this one is multiplied and finished; the time is instructions (GELU above
// all, 55 of them an element) and memory, about twice the floor of the arrays moved.  8 samples at 256^2, 32 -> 32
// channels with the spectral term: 330 us in three launches -> 52 us; 32 -> 128 with GELU: 470 -> 138 us; backward
// 128 <- 3 with GELU': 440 -> 157 us.
template <int MODE>
__global__ void __launch_bounds__(kThreads, kLayerBlocks) layer_kernel(const LayerArgs g, int* err_flag) {
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + g.o_bar);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + g.o_bar + 16);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int np = pad16(g.cout), kp = pad16(g.cin), k2p = pad16(g.k2);
  const int w_group = k_group(np);
  const int x0 = blockIdx.y * 128, tw = min(128, g.n - x0), chunks = tw / 8;
  const long long plane = static_cast<long long>(g.n) * g.n;
  const uint32_t tmem = tc_begin(mbar, 2, slot, g.cols);

  // K is padded to whole 16-wide steps with zeros on both sides; columns and rows beyond the tile
  // hold anything: they only reach products that are not stored.
  zero_smem(sm, g.o_bar);
  __syncthreads();
  for (int e = tid; e < g.cout * g.cin; e += kThreads) {
    const int co = g.w_t ? e % g.cout : e / g.cin, k = g.w_t ? e / g.cout : e % g.cin;
    *reinterpret_cast<bf16*>(sm + (k >> 3) * w_group + co * 16 + (k & 7) * 2) = g.w[e];
  }
  if (g.k2 > 0) {
    if (g.table_rows)
      copy_k_major(sm + g.o_t, k_group(128), g.table + static_cast<long long>(x0) * g.k2, g.k2, tw, g.k2 / 8);
    else
      copy_mn_major(sm + g.o_t, kMnGroup, g.table + x0, g.n, g.k2, chunks);
  }
  auto load = [&](int row, int buf) {
    const int b = row / g.n, y = row - b * g.n;
    copy_mn_major(sm + g.o_v + buf * g.v_bytes, kMnGroup,
                  g.v + static_cast<long long>(b) * g.cin * plane + static_cast<long long>(y) * g.n + x0, plane, g.cin,
                  chunks);
    if (g.k2 > 0)
      copy_k_major(sm + g.o_z + buf * g.z_bytes, w_group, g.z + (static_cast<long long>(b) * g.cout * g.n + y) * g.k2,
                   static_cast<long long>(g.n) * g.k2, g.cout, g.k2 / 8);
  };

  const int rows = g.B * g.n;
  bool ok = g.waits != 0;
  uint32_t phase = 0;
  int buf = 0;
  if (static_cast<int>(blockIdx.x) < rows) load(blockIdx.x, 0);
  cp_async_commit();
  for (int row = blockIdx.x; row < rows; row += gridDim.x, buf ^= 1) {
    if (row + static_cast<int>(gridDim.x) < rows) load(row + gridDim.x, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    fence_async_proxy();
    __syncthreads();  // every thread's copies, and its reads of the last row's accumulators
    if (tid == 0) {
      tc_fence_after();
      const uint32_t vs = smem_u32(sm + g.o_v + buf * g.v_bytes), ws = smem_u32(sm);
      const uint32_t idesc = tc_idesc(np, true, false);
      for (int s = 0; s < kp / 16; ++s)
        tc_mma(tmem, tc_smem_desc(vs + 2 * s * kMnGroup, kMnGroup, kMnChunk),
               tc_smem_desc(ws + 2 * s * w_group, w_group, 128), idesc, s > 0);
      if (g.k2 > 0) {
        const uint32_t ts = smem_u32(sm + g.o_t), zs = smem_u32(sm + g.o_z + buf * g.z_bytes);
        const uint32_t a_group = g.table_rows ? k_group(128) : kMnGroup, a_stride = g.table_rows ? 128 : kMnChunk;
        const uint32_t idesc2 = tc_idesc(np, !g.table_rows, false);
        for (int s = 0; s < k2p / 16; ++s)
          tc_mma(tmem + np, tc_smem_desc(ts + 2 * s * a_group, a_group, a_stride),
                 tc_smem_desc(zs + 2 * s * w_group, w_group, 128), idesc2, s > 0);
      }
      tc_commit(smem_u32(mbar));
    }
    const int b = row / g.n, y = row - b * g.n;
    const long long base = static_cast<long long>(b) * g.cout * plane + static_cast<long long>(y) * g.n + x0 + tid;
    const unsigned step = static_cast<unsigned>(plane);
    float next[8];
    if (MODE == 2) {
#pragma unroll
      for (int q = 0; q < 8; ++q) next[q] = tid < tw && q < g.cout ? g.pre[base + q * step] : 0.f;
    }
    if (ok) ok = mbar_wait_bounded(smem_u32(mbar), phase, kTcWaitLimit);
    phase ^= 1u;
    tc_fence_after();
    const uint32_t lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const bool valid = tid < tw && ok;
#pragma unroll 1
    for (int c0 = 0; c0 < np; c0 += 8) {
      const int count = valid ? g.cout - c0 : 0;  // channels of this chunk that are stored
      const long long o = base + c0 * plane;
      float pre[8];
      if (MODE == 2) {  // loaded a chunk ahead
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          pre[q] = next[q];
          next[q] = q + 8 < count ? g.pre[o + (q + 8) * step] : 0.f;
        }
      }
      float x[8], d[8];
      tc_ld<8>(lane + c0, x);
      if (g.k2 > 0) {
        tc_ld<8>(lane + np + c0, d);
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = __fadd_rn(x[q], d[q]);
      }
      if (g.bias) {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = __fadd_rn(x[q], c0 + q < g.cout ? __ldg(g.bias + c0 + q) : 0.f);
      }
      if (MODE == 2) {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] *= gelu_grad_f(pre[q]);
      }
      if (g.u) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < count) g.u[o + q * step] = x[q];
      }
      if (g.out) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < count) g.out[o + q * step] = __float2bfloat16_rn(MODE == 1 ? gelu_f(x[q]) : x[q]);
      }
    }
    tc_fence_before();
  }
  cp_async_wait<0>();
  tc_end(tmem, g.cols, ok, mbar + 1, err_flag);
}

// ------------------------------------------------------------------------- weight gradient
struct OuterArgs {
  const bf16* g;  // [B][cout][plane]
  const bf16* x;  // [B][cin][plane]
  float* parts;   // [B * slices][cout][cin]
  long long plane;
  int cout, cin, chunk, slices, cols, waits;
};

// parts[b, s] = sum over the `chunk` sites of slice s of g[b, :, p] x[b, :, p]^T: both operands K-major as they
// lie.  One block a slice and a serial accumulation over its slabs (the order of the sum), so the time is
// their latency unless many are in flight (STAGES slabs, most of an SM's shared memory) and then
// the instructions of a slab: 256 sites each (39 us with 64, 30 with 128) where they fit.  8 samples at 256^2: 32 x 32
// channels 208 -> 27 us, 3 x 128 240 -> 46 us, 128 x 32 416 -> 58 us.
constexpr int kOuterThreads = 256;
template <int STAGES, int LAG, int SITES>
__global__ void __launch_bounds__(kOuterThreads) outer_kernel(const OuterArgs g, int* err_flag) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ uint64_t mbar[STAGES + 1];
  __shared__ uint32_t slot;
  constexpr int kChunks = SITES / 8, kStep = kOuterThreads / kChunks;  // a thread copies every kStep-th row
  const int tid = threadIdx.x, warp = tid >> 5;
  const int mp = pad8(g.cout), np = pad16(g.cin);
  const int a_group = k_group(mp), b_group = k_group(np);
  const int a_bytes = kChunks * a_group, b_bytes = kChunks * b_group;
  unsigned char* as = sm;                       // rows beyond mp are whatever follows: never stored
  unsigned char* bs = sm + STAGES * a_bytes;
  const uint32_t tmem = tc_begin(mbar, STAGES + 1, &slot, g.cols);
  const int b = blockIdx.x / g.slices, s0 = (blockIdx.x % g.slices) * g.chunk;
  const int row0 = tid / kChunks, k0 = (tid % kChunks) * 8;
  const bf16* ga = g.g + (static_cast<long long>(b) * g.cout + row0) * g.plane + s0 + k0;
  const bf16* gb = g.x + (static_cast<long long>(b) * g.cin + row0) * g.plane + s0 + k0;
  const int dst_a = (tid % kChunks) * a_group + row0 * 16, dst_b = (tid % kChunks) * b_group + row0 * 16;
  const long long step = kStep * g.plane;
  const int slabs = (g.chunk + SITES - 1) / SITES;

  auto rows = [&](unsigned char* dst, const bf16* src, int count, bool inside) {
    if (inside) {
#pragma unroll 2
      for (int r = row0; r < count; r += kStep, dst += kStep * 16, src += step) cp_async16(dst, src);
    } else {
      for (int r = row0; r < count; r += kStep, dst += kStep * 16)
        *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
  };
  auto load = [&](int i) {
    if (i < slabs) {
      const bool inside = i * SITES + k0 < g.chunk;  // chunk is a multiple of 8
      rows(as + (i % STAGES) * a_bytes + dst_a, ga + i * SITES, g.cout, inside);
      rows(bs + (i % STAGES) * b_bytes + dst_b, gb + i * SITES, g.cin, inside);
    }
    cp_async_commit();
  };
  for (int i = 0; i < STAGES - LAG; ++i) load(i);
  const uint32_t idesc = tc_idesc(np, false, false);
  bool ok = g.waits != 0;
  for (int i = 0; i < slabs; ++i) {
    cp_async_wait<STAGES - LAG - 1>();
    fence_async_proxy();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a = smem_u32(as + (i % STAGES) * a_bytes), bb = smem_u32(bs + (i % STAGES) * b_bytes);
#pragma unroll
      for (int s = 0; s < SITES / 16; ++s)
        tc_mma(tmem, tc_smem_desc(a + 2 * s * a_group, a_group, 128),
               tc_smem_desc(bb + 2 * s * b_group, b_group, 128), idesc, i > 0 || s > 0);
      tc_commit(smem_u32(mbar + i % STAGES));
    }
    // The slot of slab i + STAGES - LAG was read by the products of slab i - LAG.
    if (i >= LAG && ok)
      ok = mbar_wait_bounded(smem_u32(mbar + (i - LAG) % STAGES), ((i - LAG) / STAGES) & 1u, kTcWaitLimit);
    load(i + STAGES - LAG);
  }
  cp_async_wait<0>();
  if (ok && slabs > 0)
    ok = mbar_wait_bounded(smem_u32(mbar + (slabs - 1) % STAGES), ((slabs - 1) / STAGES) & 1u, kTcWaitLimit);
  tc_fence_after();
  if (warp < 4) {
    const uint32_t lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    float* dst = g.parts + (static_cast<long long>(blockIdx.x) * g.cout + tid) * g.cin;
    for (int c0 = 0; c0 < np; c0 += 16) {
      float v[16];
      tc_ld<16>(lane + c0, v);
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (ok && tid < g.cout && c0 + q < g.cin) dst[c0 + q] = v[q];
    }
  }
  tc_end(tmem, g.cols, ok, mbar + STAGES, err_flag);
}

// ------------------------------------------------------------------- DFT along y, complex
struct DftYArgs {
  const bf16* gre;  // [m2][n]
  const bf16* gim;
  const bf16* s;    // [batch][K][m2], columns re | im
  float* out;       // [batch][M][m2] or null
  bf16* out_bf;
  int n, m2, K, M, cols, o_s, o_bar, waits;
  float sign;       // of gim's product in the real part
};

// out = G s (INVERSE: G^H s) for the complex matrix of one (sample, channel): with D1 = Gre s and D2 = Gim s over
// re and im columns together, re = D1_re + sign D2_im, im = D1_im - sign D2_re.  One launch in place of four
// general GEMMs with FP32 products read and added between them; the problem is a few KB a block, so
// its time is one round of copies and one of products.  256 matrices, n = 256, 16 modes: 80 and
// 100 us in four launches each -> 13 and 12 us.
template <bool INVERSE>
__global__ void __launch_bounds__(kThreads) dft_y_kernel(const DftYArgs g, int* err_flag) {
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + g.o_bar);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + g.o_bar + 16);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int kp = pad16(g.K), np = pad16(g.m2);
  const int a_group = INVERSE ? kMnGroup : k_group(g.m2);
  const int a_stride = INVERSE ? kMnChunk : 128;
  const int a_bytes = (kp / 8) * a_group;
  const int s_chunks = g.m2 / 8, b_group = (np / 8) * kMnChunk;
  const int m0 = blockIdx.y * 128, tm = min(128, g.M - m0);
  const uint32_t tmem = tc_begin(mbar, 2, slot, g.cols);
  if (kp != g.K || np != g.m2) {
    zero_smem(sm, g.o_bar);
    __syncthreads();
  }
  for (int h = 0; h < 2; ++h) {
    const bf16* G = h ? g.gim : g.gre;
    unsigned char* a = sm + h * a_bytes;
    if (INVERSE)  // A = G^T: rows y, k = the kept frequencies, M-major
      copy_mn_major(a, kMnGroup, G + m0, g.n, g.K, tm / 8);
    else
      copy_k_major(a, a_group, G, g.n, g.m2, g.K / 8);
  }
  copy_mn_major(sm + g.o_s, b_group, g.s + static_cast<long long>(blockIdx.x) * g.K * g.m2, g.m2, g.K, s_chunks);
  cp_async_commit();
  cp_async_wait<0>();
  fence_async_proxy();
  __syncthreads();
  if (tid == 0) {
    tc_fence_after();
    const uint32_t idesc = tc_idesc(np, INVERSE, true);
    const uint32_t b = smem_u32(sm + g.o_s);
    for (int h = 0; h < 2; ++h) {
      const uint32_t a = smem_u32(sm + h * a_bytes);
      for (int s = 0; s < kp / 16; ++s)
        tc_mma(tmem + h * np, tc_smem_desc(a + 2 * s * a_group, a_group, a_stride),
               tc_smem_desc(b + 2 * s * b_group, b_group, kMnChunk), idesc, s > 0);
    }
    tc_commit(smem_u32(mbar));
  }
  const bool ok = g.waits && mbar_wait_bounded(smem_u32(mbar), 0u, kTcWaitLimit);
  tc_fence_after();
  const uint32_t lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  const int m = g.m2 / 2;
  const long long o = (static_cast<long long>(blockIdx.x) * g.M + m0 + tid) * g.m2;
  for (int c = 0; c < m; c += 4) {
    float r1[4], i1[4], r2[4], i2[4];
    tc_ld<4>(lane + c, r1);
    tc_ld<4>(lane + m + c, i1);
    tc_ld<4>(lane + np + c, r2);
    tc_ld<4>(lane + np + m + c, i2);
    if (!ok || tid >= tm) continue;
    float re[4], im[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      re[q] = __fadd_rn(r1[q], g.sign * i2[q]);
      im[q] = __fadd_rn(i1[q], -g.sign * r2[q]);
    }
    if (g.out) {
      *reinterpret_cast<float4*>(g.out + o + c) = make_float4(re[0], re[1], re[2], re[3]);
      *reinterpret_cast<float4*>(g.out + o + m + c) = make_float4(im[0], im[1], im[2], im[3]);
    }
    if (g.out_bf) {
      __nv_bfloat162 p[4] = {__floats2bfloat162_rn(re[0], re[1]), __floats2bfloat162_rn(re[2], re[3]),
                             __floats2bfloat162_rn(im[0], im[1]), __floats2bfloat162_rn(im[2], im[3])};
      *reinterpret_cast<uint2*>(g.out_bf + o + c) = *reinterpret_cast<uint2*>(p);
      *reinterpret_cast<uint2*>(g.out_bf + o + m + c) = *reinterpret_cast<uint2*>(p + 2);
    }
  }
  tc_end(tmem, g.cols, ok, mbar + 1, err_flag);
}

// ------------------------------------------------------------------------ DFT along x, rows
struct DftXArgs {
  const bf16* v;      // [rows][n]
  const bf16* table;  // [n][m2], or [m2][n] when table_rows
  bf16* out;          // [rows][m2]
  long long rows;
  int n, m2, table_rows, cols, o_b, o_bar, waits;
};

// out = v T, rounded to BF16: 128 rows a block, all of their n values in flight at once, and a second
// block on the SM copies meanwhile.  65536 rows of 256 values, 32 columns: 33 (and 9 to round) -> 21 us.
__global__ void __launch_bounds__(kThreads) dft_x_kernel(const DftXArgs g, int* err_flag) {
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + g.o_bar);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + g.o_bar + 16);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int kp = pad16(g.n), np = pad16(g.m2);
  const int b_group = g.table_rows ? k_group(np) : (np / 8) * kMnChunk;
  const long long r0 = static_cast<long long>(blockIdx.x) * 128;
  const int tm = static_cast<int>(g.rows - r0 < 128 ? g.rows - r0 : 128);
  const uint32_t tmem = tc_begin(mbar, 2, slot, g.cols);
  if (kp != g.n) {  // one group of 8 zeros on both sides
    zero_smem(sm + (kp / 8 - 1) * k_group(128), k_group(128));
    zero_smem(sm + g.o_b + (kp / 8 - 1) * b_group, b_group);
    __syncthreads();
  }
  copy_k_major(sm, k_group(128), g.v + r0 * g.n, g.n, tm, g.n / 8);
  if (g.table_rows)
    copy_k_major(sm + g.o_b, b_group, g.table, g.n, g.m2, g.n / 8);
  else
    copy_mn_major(sm + g.o_b, b_group, g.table, g.m2, g.n, g.m2 / 8);
  cp_async_commit();
  cp_async_wait<0>();
  fence_async_proxy();
  __syncthreads();
  if (tid == 0) {
    tc_fence_after();
    const uint32_t a = smem_u32(sm), b = smem_u32(sm + g.o_b);
    const uint32_t idesc = tc_idesc(np, false, !g.table_rows);
    for (int s = 0; s < kp / 16; ++s)
      tc_mma(tmem, tc_smem_desc(a + 2 * s * k_group(128), k_group(128), 128),
             tc_smem_desc(b + 2 * s * b_group, b_group, g.table_rows ? 128 : kMnChunk), idesc, s > 0);
    tc_commit(smem_u32(mbar));
  }
  const bool ok = g.waits && mbar_wait_bounded(smem_u32(mbar), 0u, kTcWaitLimit);
  tc_fence_after();
  const uint32_t lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  bf16* dst = g.out + (r0 + tid) * g.m2;
  for (int c = 0; c < g.m2; c += 8) {
    float v[8];
    tc_ld<8>(lane + c, v);
    if (!ok || tid >= tm) continue;
    __nv_bfloat162 p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
    *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<uint4*>(p);
  }
  tc_end(tmem, g.cols, ok, mbar + 1, err_flag);
}

// ------------------------------------------------------------------------------ geometry
int tmem_cols(int need) {
  int c = 32;
  while (c < need) c *= 2;
  return c;
}

// Shared memory to ask for: no more blocks on an SM than its 512 TMEM columns serve.
int block_smem(int need, int cols) {
  const int blocks = 512 / cols;
  return std::max(need, kMaxSmem / (blocks + 1) + 16);
}

int layer_geometry(LayerArgs* a) {
  const int kp = pad16(a->cin), np = pad16(a->cout), k2p = pad16(a->k2);
  a->o_t = (kp / 8) * k_group(np);
  a->o_v = a->o_t + (k2p / 8) * (a->table_rows ? k_group(128) : kMnGroup);
  a->v_bytes = (kp / 8) * kMnGroup;
  a->o_z = a->o_v + 2 * a->v_bytes;
  a->z_bytes = (k2p / 8) * k_group(np);
  a->o_bar = a->o_z + 2 * a->z_bytes;
  a->cols = tmem_cols(np * (a->k2 > 0 ? 2 : 1));
  return block_smem(a->o_bar + 32, a->cols);
}

template <bool INVERSE>
int dft_y_geometry(DftYArgs* a) {
  const int kp = pad16(a->K), np = pad16(a->m2);
  a->o_s = 2 * (kp / 8) * (INVERSE ? kMnGroup : k_group(a->m2));
  // The forward A operand has m2 rows: the 128-row products read up to 2 KB past its last group,
  // which the s operand and the barrier's area cover.
  a->o_bar = a->o_s + std::max(2048, (kp / 8) * (np / 8) * kMnChunk);
  a->cols = tmem_cols(2 * np);
  return block_smem(a->o_bar + 32, a->cols);
}

int dft_x_geometry(DftXArgs* a) {
  const int kp = pad16(a->n), np = pad16(a->m2);
  a->o_b = (kp / 8) * k_group(128);
  a->o_bar = a->o_b + (kp / 8) * (a->table_rows ? k_group(np) : (np / 8) * kMnChunk);
  a->cols = tmem_cols(np);
  return block_smem(a->o_bar + 32, a->cols);
}

int outer_bytes(int cout, int cin) { return 16 * (k_group(pad8(cout)) + k_group(pad16(cin))); }

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 152;
  return sms;
}

template <bool INVERSE>
int run_dft_y(const pg::DftYArgs& in, int batch, cudaStream_t stream) {
  DftYArgs a = in;
  const int smem = dft_y_geometry<INVERSE>(&a);
  PG_CHECK(smem <= kMaxSmem, PG_ERR_UNSUPPORTED, "pg_fno_dft_y: does not fit shared memory");
  int* flag = nullptr;
  PG_CUDA(gemm_timeout_flag(&flag));
  PG_CUDA(allow_smem(dft_y_kernel<INVERSE>));
  dft_y_kernel<INVERSE><<<dim3(batch, (a.M + 127) / 128), kThreads, smem, stream>>>(a, flag);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

}  // namespace
}  // namespace pg

extern "C" {

// Whether the fused kernels serve a network on n x n sites: 16-byte rows (n and 2 modes multiples of
// 8), channels within one tile, operands within an SM's shared memory, and tcgen05 as the GEMM engine.
int pg_fno_fused(int32_t n, int32_t modes, int32_t max_channels, int32_t* fused) {
  PG_CHECK(fused, PG_ERR_INVALID, "pg_fno_fused: null argument");
  *fused = 0;
  if (pg::gemm_engine() != 0 || n < 8 || n % 8 != 0 || modes < 4 || modes % 4 != 0 || modes > 64) return PG_OK;
  if (max_channels < 1 || max_channels > 128) return PG_OK;
  pg::LayerArgs l{};
  l.cin = l.cout = max_channels;
  l.k2 = 2 * modes;
  pg::DftYArgs y{};
  y.K = n;
  y.m2 = 2 * modes;
  pg::DftXArgs x{};
  x.n = n;
  x.m2 = 2 * modes;
  int smem = std::max(pg::dft_y_geometry<false>(&y), pg::dft_x_geometry(&x));
  x.table_rows = 1;
  smem = std::max(smem, std::max(pg::dft_x_geometry(&x), pg::layer_geometry(&l)));
  y.K = 2 * modes;
  smem = std::max(smem, pg::dft_y_geometry<true>(&y));
  *fused = smem <= pg::kMaxSmem && l.cols <= 512 ? 1 : 0;
  return PG_OK;
}

int pg_fno_layer(const void* w, int32_t w_transposed, const void* v, const void* z, const void* table,
                 int32_t table_rows, const float* bias, const float* pre, float* u, void* out_bf16,
                 int32_t B, int32_t cin, int32_t cout, int32_t n, int32_t modes2, int32_t mode, void* stream) {
  PG_CHECK(w && v && (u || out_bf16) && B > 0 && cin > 0 && cout > 0 && n > 0, PG_ERR_INVALID,
           "pg_fno_layer: bad argument");
  PG_CHECK(cin <= 128 && cout <= 128 && n % 8 == 0 && modes2 >= 0 && modes2 % 8 == 0 && mode >= 0 && mode <= 2,
           PG_ERR_UNSUPPORTED, "pg_fno_layer: sizes");
  PG_CHECK((modes2 == 0 || (z && table)) && (mode != 2 || pre), PG_ERR_INVALID, "pg_fno_layer: null operand");
  PG_CHECK(pg::aligned16(v) && pg::aligned16(z) && pg::aligned16(table), PG_ERR_INVALID,
           "pg_fno_layer: operands must start on 16-byte boundaries");
  pg::LayerArgs a{};
  a.w = static_cast<const __nv_bfloat16*>(w);
  a.v = static_cast<const __nv_bfloat16*>(v);
  a.z = static_cast<const __nv_bfloat16*>(z);
  a.table = static_cast<const __nv_bfloat16*>(table);
  a.bias = bias;
  a.pre = pre;
  a.u = u;
  a.out = static_cast<__nv_bfloat16*>(out_bf16);
  a.w_t = w_transposed ? 1 : 0;
  a.table_rows = table_rows ? 1 : 0;
  a.cin = cin;
  a.cout = cout;
  a.n = n;
  a.B = B;
  a.k2 = modes2;
  a.waits = pg::gemm_wait_limit() > 0;
  const int smem = pg::layer_geometry(&a);
  PG_CHECK(smem <= pg::kMaxSmem && a.cols <= 512, PG_ERR_UNSUPPORTED, "pg_fno_layer: does not fit an SM");
  int* flag = nullptr;
  PG_CUDA(pg::gemm_timeout_flag(&flag));
  auto kernel = mode == 2 ? pg::layer_kernel<2> : mode == 1 ? pg::layer_kernel<1> : pg::layer_kernel<0>;
  PG_CUDA(pg::allow_smem(kernel));
  const int per_sm = std::min({pg::kLayerBlocks, 512 / a.cols, 228 * 1024 / (smem + 1024)});
  const int tiles = (n + 127) / 128;
  const int resident = std::max(1, per_sm * pg::sm_count() / tiles);
  kernel<<<dim3(std::min(B * n, resident), tiles), pg::kThreads, smem,
                     static_cast<cudaStream_t>(stream)>>>(a, flag);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

int pg_fno_outer(const void* g, const void* x, float* parts, int32_t B, int32_t cout, int32_t cin, int64_t plane,
                 int32_t slices, void* stream) {
  PG_CHECK(g && x && parts && B > 0 && cout > 0 && cin > 0 && plane > 0 && slices > 0, PG_ERR_INVALID,
           "pg_fno_outer: bad argument");
  PG_CHECK(cin <= 128 && cout <= 128 && plane % (8LL * slices) == 0 && plane < (1LL << 31), PG_ERR_UNSUPPORTED,
           "pg_fno_outer: sizes");
  PG_CHECK(pg::aligned16(g) && pg::aligned16(x), PG_ERR_INVALID,
           "pg_fno_outer: operands must start on 16-byte boundaries");
  pg::OuterArgs a{};
  a.g = static_cast<const __nv_bfloat16*>(g);
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.parts = parts;
  a.plane = plane;
  a.cout = cout;
  a.cin = cin;
  a.slices = slices;
  a.chunk = static_cast<int>(plane / slices);
  a.cols = pg::tmem_cols(pg::pad16(cin));
  a.waits = pg::gemm_wait_limit() > 0;
  int* flag = nullptr;
  PG_CUDA(pg::gemm_timeout_flag(&flag));
  const int stage = pg::outer_bytes(cout, cin);  // of 128 sites
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // 2 KB past the stages: the 128-row products read that far beyond the last rows of A.
  const int blocks = B * slices;
  auto run = [&](auto kernel, int slabs) {
    const int smem = pg::block_smem(slabs * stage + 2048, a.cols);
    const cudaError_t e = pg::allow_smem(kernel, 1024);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, pg::kOuterThreads, smem, st>>>(a, flag);
    return cudaGetLastError();
  };
  constexpr int room = 220 * 1024 - 2048;
  if (10 * stage <= room)
    PG_CUDA(run(pg::outer_kernel<5, 2, 256>, 10));
  else if (5 * stage <= room)
    PG_CUDA(run(pg::outer_kernel<5, 2, 128>, 5));
  else
    PG_CUDA(run(pg::outer_kernel<3, 1, 128>, 3));
  return PG_OK;
}

int pg_fno_dft_y(const void* gre, const void* gim, const void* s, float* out, void* out_bf16, int32_t batch,
                 int32_t n, int32_t modes, int32_t inverse, void* stream) {
  PG_CHECK(gre && gim && s && (out || out_bf16) && batch > 0 && n > 0 && modes > 0, PG_ERR_INVALID,
           "pg_fno_dft_y: bad argument");
  PG_CHECK(n % 8 == 0 && modes % 4 == 0 && modes <= 64, PG_ERR_UNSUPPORTED, "pg_fno_dft_y: sizes");
  PG_CHECK(pg::aligned16(gre) && pg::aligned16(gim) && pg::aligned16(s) && pg::aligned16(out) &&
               pg::aligned16(out_bf16),
           PG_ERR_INVALID, "pg_fno_dft_y: arrays must start on 16-byte boundaries");
  pg::DftYArgs a{};
  a.gre = static_cast<const __nv_bfloat16*>(gre);
  a.gim = static_cast<const __nv_bfloat16*>(gim);
  a.s = static_cast<const __nv_bfloat16*>(s);
  a.out = out;
  a.out_bf = static_cast<__nv_bfloat16*>(out_bf16);
  a.n = n;
  a.m2 = 2 * modes;
  a.K = inverse ? 2 * modes : n;
  a.M = inverse ? n : 2 * modes;
  a.sign = inverse ? 1.f : -1.f;
  a.waits = pg::gemm_wait_limit() > 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return inverse ? pg::run_dft_y<true>(a, batch, st) : pg::run_dft_y<false>(a, batch, st);
}

int pg_fno_dft_x(const void* v, const void* table, int32_t table_rows, void* out_bf16, int64_t rows, int32_t n,
                 int32_t modes, void* stream) {
  PG_CHECK(v && table && out_bf16 && rows > 0 && n > 0 && modes > 0, PG_ERR_INVALID, "pg_fno_dft_x: bad argument");
  PG_CHECK(n % 8 == 0 && modes % 4 == 0 && modes <= 64 && (rows + 127) / 128 < (1LL << 31), PG_ERR_UNSUPPORTED,
           "pg_fno_dft_x: sizes");
  PG_CHECK(pg::aligned16(v) && pg::aligned16(table) && pg::aligned16(out_bf16), PG_ERR_INVALID,
           "pg_fno_dft_x: arrays must start on 16-byte boundaries");
  pg::DftXArgs a{};
  a.v = static_cast<const __nv_bfloat16*>(v);
  a.table = static_cast<const __nv_bfloat16*>(table);
  a.out = static_cast<__nv_bfloat16*>(out_bf16);
  a.rows = rows;
  a.n = n;
  a.m2 = 2 * modes;
  a.table_rows = table_rows ? 1 : 0;
  a.waits = pg::gemm_wait_limit() > 0;
  const int smem = pg::dft_x_geometry(&a);
  PG_CHECK(smem <= pg::kMaxSmem, PG_ERR_UNSUPPORTED, "pg_fno_dft_x: does not fit shared memory");
  int* flag = nullptr;
  PG_CUDA(pg::gemm_timeout_flag(&flag));
  PG_CUDA(pg::allow_smem(pg::dft_x_kernel));
  pg::dft_x_kernel<<<static_cast<unsigned>((rows + 127) / 128), pg::kThreads, smem,
                     static_cast<cudaStream_t>(stream)>>>(a, flag);
  PG_CUDA(cudaGetLastError());
  return PG_OK;
}

}  // extern "C"
