// IFRK column pass for FP32 columns of 1024 sites of a one-component field with one single
// reservoir and one laser: register-resident four-step FFTs with 32 values a thread.
//
// A 1024-point transform is 1024 = 32 x 32 (n = n2 + 32 n1, k = k1 + 32 k2):
//   X[k1 + 32 k2] = sum_n2 W_32^{n2 k2} W_1024^{n2 k1} sum_n1 x[n2 + 32 n1] W_32^{n1 k1}.
// A thread holds the 32 values x[n2 + 32 n1] of its n2 (n1 = register index), does the inner
// 32-point DFT in registers, multiplies by W_1024^{n2 k1}, exchanges once through shared memory so
// that it holds the 32 values of one k1, and does the outer 32-point DFT: it ends with
// X[k1 + 32 k2] (k2 = register index), the layout it started from.  A block takes a panel of
// eight columns (thread = (column, n2)); between the inverse and forward transforms the site
// step (ifrk_sites.cuh) runs over the panel in shared memory.
//
// Why this pass beside ifrk_reg.cu's: its site step has up to seven loads a site and little
// arithmetic, so it is bound by loads in flight; 128 registers a thread hold batches of eight
// sites unspilled, 64 hold two.  A fixed step of 8 x 1024^2 takes 913 us with this column pass and
// 1041 with the sixteen-value one, of 1024^2 x 1 164 against 179.  (The split-step column pass,
// bound by its arithmetic, is faster on sixteen values.)
//
// Precision: every twiddle that is not +-1 or +-i is applied as a rounded value plus its
// remainder (the 32-point constants and the table W_1024^{n2 k1}).
#include <cmath>

#include "ifrk_internal.h"
#include "ifrk_sites.cuh"
#include "split_local.cuh"

namespace pg {
namespace {

constexpr int kN = 1024;
constexpr int kPanel = 8;                   // columns a block (column pass)
constexpr int kXStride = 33;                // padded row of the 32 x 32 exchange
constexpr int kPanelStride = 32 * 33 + 4;   // one column's exchange block (elements = 4 mod 16)

// W_32^e = exp(-2 pi i e / 32) = c - i s for e = 1..15 (not 8) as {c, s} rounded to FP32 and
// the remainders {c - c_fp32, s - s_fp32}, from the double-precision cos and sin; e is a
// constant once the DFT loops are unrolled, so the switch folds to immediates.
__device__ __forceinline__ float4 w32(int e) {
  switch (e) {
    case 1: return make_float4(0.9807852506637573f, 0.19509032368659973f, 2.9739473106360492e-08f, -1.6704715388726754e-09f);
    case 2: return make_float4(0.9238795042037964f, 0.3826834261417389f, 2.830748968563057e-08f, 6.2233507236442165e-09f);
    case 3: return make_float4(0.8314695954322815f, 0.5555702447891235f, 1.687026340846387e-08f, -1.1769521357507529e-08f);
    case 4: return make_float4(0.7071067690849304f, 0.7071067690849304f, 1.2101617485882343e-08f, 1.2101617485882343e-08f);
    case 5: return make_float4(0.5555702447891235f, 0.8314695954322815f, -1.1769521357507529e-08f, 1.687026340846387e-08f);
    case 6: return make_float4(0.3826834261417389f, 0.9238795042037964f, 6.2233507236442165e-09f, 2.830748968563057e-08f);
    case 7: return make_float4(0.19509032368659973f, 0.9807852506637573f, -1.670471427850373e-09f, 2.9739473106360492e-08f);
    case 9: return make_float4(-0.19509032368659973f, 0.9807852506637573f, 1.6704715388726754e-09f, 2.9739473106360492e-08f);
    case 10: return make_float4(-0.3826834261417389f, 0.9238795042037964f, -6.2233507236442165e-09f, 2.830748968563057e-08f);
    case 11: return make_float4(-0.5555702447891235f, 0.8314695954322815f, 1.1769521357507529e-08f, 1.687026340846387e-08f);
    case 12: return make_float4(-0.7071067690849304f, 0.7071067690849304f, -1.2101617485882343e-08f, 1.2101617485882343e-08f);
    case 13: return make_float4(-0.8314695954322815f, 0.5555702447891235f, -1.687026340846387e-08f, -1.1769521357507529e-08f);
    case 14: return make_float4(-0.9238795042037964f, 0.3826834261417389f, -2.830748968563057e-08f, 6.223351167733426e-09f);
    case 15: return make_float4(-0.9807852506637573f, 0.19509032368659973f, -2.9739473106360492e-08f, -1.6704710947834656e-09f);
    default: return make_float4(1.0f, 0.0f, 0.0f, 0.0f);
  }
}

__host__ __device__ constexpr int brev5(int i) {
  return ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
}

// x * W_32^e (forward) or x * conj(W_32^e) (inverse); e is a constant once unrolled.
template <bool INV>
__device__ __forceinline__ float2 w32mul(float2 x, int e) {
  if (e == 0) return x;
  if (e == 8) return INV ? make_float2(-x.y, x.x) : make_float2(x.y, -x.x);
  const float4 w = w32(e);
  const float ch = w.x, sh = w.y, cl = w.z, sl = w.w;
  // forward: (x.x c + x.y s) + i (x.y c - x.x s); inverse: (x.x c - x.y s) + i (x.y c + x.x s)
  const float ys = INV ? -x.y : x.y;
  const float xs = INV ? x.x : -x.x;
  const float re = fmaf(x.x, ch, fmaf(ys, sh, fmaf(x.x, cl, ys * sl)));
  const float im = fmaf(x.y, ch, fmaf(xs, sh, fmaf(x.y, cl, xs * sl)));
  return make_float2(re, im);
}

// In-register 32-point DFT (radix 2, decimation in time; the bit-reversed read is a renaming).
template <bool INV>
__device__ __forceinline__ void dft32(float2 (&v)[32]) {
  float2 a[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = v[brev5(i)];
#pragma unroll
  for (int s = 1; s <= 5; ++s) {
#pragma unroll
    for (int b = 0; b < 16; ++b) {  // the 16 butterflies of stage s (span m = 2^s)
      const int h = 1 << (s - 1);
      const int j = b & (h - 1);
      const int lo = ((b >> (s - 1)) << s) + j;
      const float2 u = a[lo];
      const float2 t = w32mul<INV>(a[lo + h], j << (5 - s));
      a[lo] = make_float2(u.x + t.x, u.y + t.y);
      a[lo + h] = make_float2(u.x - t.x, u.y - t.y);
    }
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = a[i];
}

// conj of the 32 values: an inverse transform is the forward transform of the conjugate,
// conjugated, so each kernel carries one copy of the transform's code (an instruction-cache
// working set half as large; the kernels were stalled on instruction fetch).
__device__ __forceinline__ void conj32(float2 (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i].y = -v[i].y;
}

// Inner DFT and the W_1024^{n2 k1} factors (tw4[k1][n2]: rounded value and remainder).
template <bool INV>
__device__ __forceinline__ void four_step_first(float2 (&v)[32], int n2, const float4* tw4) {
  dft32<INV>(v);
#pragma unroll
  for (int k1 = 1; k1 < 32; ++k1) {
    const float4 w = tw4[k1 * 32 + n2];
    v[k1] = INV ? cmulc2f(v[k1], make_float2(w.x, w.y), make_float2(w.z, w.w))
                : cmul2f(v[k1], make_float2(w.x, w.y), make_float2(w.z, w.w));
  }
}

// ------------------------------------------------------------------ column pass
// A forward 1024-point transform of the block's eight columns (thread = (column c, n2 = p));
// pan is the panel's exchange buffer ([c][k1][n2], columns kPanelStride apart).
__device__ __forceinline__ void fft1024_panel(float2 (&v)[32], int p, int c, float2* pan,
                                              const float4* tw4) {
  four_step_first<false>(v, p, tw4);
  __syncthreads();  // every earlier read of pan is done
#pragma unroll
  for (int k1 = 0; k1 < 32; ++k1) pan[c * kPanelStride + k1 * kXStride + p] = v[k1];
  __syncthreads();
#pragma unroll
  for (int n2 = 0; n2 < 32; ++n2) v[n2] = pan[c * kPanelStride + p * kXStride + n2];
  dft32<false>(v);
}

// ------------------------------------------------------------------ IFRK column pass
// ifrk_col_kernel (ifrk.cu) for FP32 columns of 1024 sites of a one-component field: the
// forward-only pass that forms W (mode 3, any reservoir), and the stage and step-end passes
// (modes 0 and 1) for one single reservoir and one laser (ifrk_sites_batched).  An eight-column
// panel, the inverse transform, the site step over the panel in shared memory in site order
// (ifrk_sites.cuh, kIfrkBatch sites a thread at a stage, kIfrkEndBatch at the step end), the
// forward transform.  The error norm (mode 2) stays on the generic pass.
constexpr int kIfrkBatch = 8;     // 4 / 2 measured 4 % slower
constexpr int kIfrkEndBatch = 4;
__global__ void __launch_bounds__(kPanel * 32, 2)
    ifrk_col_fast_kernel(float2* __restrict__ psi, const float* __restrict__ n0,
                         float* __restrict__ dn_out, float* __restrict__ n_out,
                         float2* __restrict__ psi_start, float2* __restrict__ psi_new,
                         const float* __restrict__ pump, const float* __restrict__ potential,
                         const float4* __restrict__ tw4_g,
                         const SplitConst<float>* __restrict__ consts,
                         const float* __restrict__ scales,
                         const unsigned long long* __restrict__ step_base, const IfrkColArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // The twiddle table is read through L1 rather than staged in shared memory: two blocks an
  // SM then leave the driver a larger L1 for the site step's loads (+4.5 % on the step; the
  // split-step column pass, with fewer loads a site, gains nothing from it).
  const float4* tw4 = tw4_g;                          // [32][32]
  float2* pan = reinterpret_cast<float2*>(smem_raw);  // exchange, or [row][c] for the site step
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = lane & (kPanel - 1);
  const int p = warp * 4 + (lane >> 3);  // n2: 0..31
  const int member = blockIdx.z;
  const int x0 = blockIdx.x * kPanel;
  const long long plane = static_cast<long long>(a.nx) * kN;
  float2* d = psi + member * plane + x0 + c;
  float2 v[32];
#pragma unroll
  for (int t = 0; t < 32; ++t) v[t] = d[static_cast<long long>(p + 32 * t) * a.nx];
  // Phase 0: the inverse transform (conj32 around the forward one) and the site step;
  // phase 1: the forward transform (one copy of the transform's code).
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.inverse : a.forward) {
      if (ph == 0) conj32(v);
      fft1024_panel(v, p, c, pan, tw4);
      if (ph == 0) conj32(v);
    }
    if (ph == 1 || a.mode == 3) continue;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 32; ++t) pan[(p + 32 * t) * kPanel + c] = v[t];
    __syncthreads();
    {
      const SplitConst<float> k = consts[member];
      const float s0 = scales ? scales[static_cast<long long>(a.scale_index) * a.members + member]
                              : 0.f;
      const float* pm = pump + member * a.pump_stride;
      const float* vm =
          potential ? potential + member * a.pot_stride * (a.potential == 2 ? 2 : 1) : nullptr;
      const unsigned long long step = a.noise ? step_base[0] + a.step_offset : 0ull;
      const PhiloxCellPrefix prefix = philox_cell_prefix(
          static_cast<uint32_t>(step), static_cast<uint32_t>(step >> 32), 1u,
          static_cast<uint32_t>(k.seed), static_cast<uint32_t>(k.seed >> 32));
      ifrk_sites_run<float, kIfrkBatch, kIfrkEndBatch>(pan, PanelSites{kPanel, 3, a.nx, x0, kPanel * kN}, a,
                                                       k, member * plane, n0, dn_out, n_out,
                                                       psi_start, psi_new, pm, vm, s0, prefix);
    }
    __syncthreads();
    if (a.mode == 1 && !a.forward) return;
#pragma unroll
    for (int t = 0; t < 32; ++t) v[t] = pan[(p + 32 * t) * kPanel + c];
  }
#pragma unroll
  for (int t = 0; t < 32; ++t) d[static_cast<long long>(p + 32 * t) * a.nx] = v[t];
}

size_t ifrk_col_fast_smem() { return kPanel * kPanelStride * sizeof(float2); }

}  // namespace

bool ifrk_col_fast_size(int nx, int ny) { return ny == kN && nx % kPanel == 0; }

void ifrk_col_fast_twiddles(float* out) {
  // tw4[k1][n2] = W_1024^{n2 k1}: rounded value and remainder, from double precision.
  const double pi = 3.141592653589793238462643383279502884;
  for (int k1 = 0; k1 < 32; ++k1)
    for (int n2 = 0; n2 < 32; ++n2) {
      const double ang = -2.0 * pi * static_cast<double>((n2 * k1) % kN) / kN;
      const double cr = std::cos(ang), ci = std::sin(ang);
      float* o = out + 4 * (k1 * 32 + n2);
      o[0] = static_cast<float>(cr);
      o[1] = static_cast<float>(ci);
      o[2] = static_cast<float>(cr - static_cast<double>(o[0]));
      o[3] = static_cast<float>(ci - static_cast<double>(o[1]));
    }
}

cudaError_t configure_ifrk_col_fast() {
  return cudaFuncSetAttribute(ifrk_col_fast_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(ifrk_col_fast_smem()));
}

bool ifrk_fast_col(const IfrkColArgs& a) {
  return a.comps == 1 && a.ny == kN && a.nx % kPanel == 0 &&
         static_cast<long long>(a.nx) * kN <= 0x7fffffffLL &&
         (a.mode == 3 || ifrk_sites_batched(a));
}

cudaError_t launch_ifrk_col_fast(float* psi, const float* n0, float* dn_out, float* n_out,
                                 const float* psi_start, const float* psi_new, const float* pump,
                                 const float* potential, const float* tw4,
                                 const SplitConst<float>* consts, const float* scales,
                                 const unsigned long long* step_base, const IfrkColArgs& a,
                                 cudaStream_t stream) {
  const dim3 grid(a.nx / kPanel, 1, a.members);
  ifrk_col_fast_kernel<<<grid, kPanel * 32, ifrk_col_fast_smem(), stream>>>(
      reinterpret_cast<float2*>(psi), n0, dn_out, n_out,
      reinterpret_cast<float2*>(const_cast<float*>(psi_start)),
      reinterpret_cast<float2*>(const_cast<float*>(psi_new)), pump, potential,
      reinterpret_cast<const float4*>(tw4), consts, scales, step_base, a);
  return cudaGetLastError();
}

}  // namespace pg
