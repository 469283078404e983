// Register-resident FP32 FFTs of 64 to 4096 points, V = 16 (to 512 points, 8) values a thread
// (device code of the split-step and IFRK passes).
//
// N = V x V x L.  Thread t of a transform's M = N / V holds x[t + M m], m < V:
//   pass 1  a V-point DFT over m gives k1; times W_N^{t k1}; exchange;
//   pass 2  thread (q = t mod V, u = t / V) takes the V values of sequence k1 = q at positions
//           u + L m: a V-point DFT gives j1; times W_M^{u j1}; exchange;
//   last    thread t takes, for each of its groups g = k1 + V j1 = t + M i, the L values of u: an
//           L-point DFT gives j2.
// The result X[g + V^2 j2] is again X[t + M m]: a transform ends in the layout it starts from, so
// a pass over the grid loads its values once, transforms, works on them and transforms back
// without leaving the registers but for the exchanges (one at V^2 points, two above; the
// shared-memory Stockham passes of fft.cuh make four to six, each behind two barriers).  Both
// exchanges write and read the buffer at base + m * stride, so both DFT passes run the same code
// (one copy: 32 values a thread with straight-line 32-point transforms stalled on instruction
// fetch).  Sixteen values a thread need 64 registers, so 32 warps an SM cover the loads
// of the site steps between the transforms; eight put twice the threads on a small grid, whose
// time is that of one thread's chain.
//
// Precision: every factor that is not +-1 or +-i is applied as a rounded value plus its remainder:
// rounded factors alone carry a per-step amplitude bias that drifts the norm over long runs.
#pragma once
#include "fft.cuh"

namespace pg {
namespace {

template <int N, int V>
struct RegFft {
  static_assert(N >= V * V, "two V-point passes");
  static constexpr int M = N / V;         // threads of one transform
  static constexpr int L = N / (V * V);   // points of the last DFT
  static constexpr int Mp = M + 1;        // padded sequence of the first exchange
  static constexpr int SLOTS = V * Mp;    // values of one transform's exchange buffer
};

// --- complex arithmetic: packed FP32x2 where no halves swap ------------------------------------
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
// a - i b and a + i b
__device__ __forceinline__ float2 csub_i(float2 a, float2 b) { return float2{a.x + b.y, a.y - b.x}; }
__device__ __forceinline__ float2 cadd_i(float2 a, float2 b) { return float2{a.x - b.y, a.y + b.x}; }

// x times the real constant h + l, rounded value and remainder.
__device__ __forceinline__ float rmul(float x, float h, float l) { return fmaf(x, h, x * l); }
// x (c - i s) with constants c = ch + cl, s = sh + sl.
__device__ __forceinline__ float2 cmul_const(float2 x, float ch, float cl, float sh, float sl) {
  return make_float2(fmaf(x.x, ch, fmaf(x.y, sh, fmaf(x.x, cl, x.y * sl))),
                     fmaf(x.y, ch, fmaf(-x.x, sh, fmaf(x.y, cl, -x.x * sl))));
}

// cos and sin of pi / 8 and sqrt(1/2) in double precision, split at compile time.
struct DftConst {
  static constexpr double kC8 = 0.92387953251128675613, kS8 = 0.38268343236508977173,
                          kR = 0.70710678118654752440;
  static constexpr float ch = static_cast<float>(kC8), cl = static_cast<float>(kC8 - static_cast<double>(ch));
  static constexpr float sh = static_cast<float>(kS8), sl = static_cast<float>(kS8 - static_cast<double>(sh));
  static constexpr float rh = static_cast<float>(kR), rl = static_cast<float>(kR - static_cast<double>(rh));
};

// x W_8 = x (1 - i) / sqrt 2 and x W_8^3 = x (-1 - i) / sqrt 2.
__device__ __forceinline__ float2 mul_w8(float2 x) {
  using K = DftConst;
  return float2{rmul(x.x + x.y, K::rh, K::rl), rmul(x.y - x.x, K::rh, K::rl)};
}
__device__ __forceinline__ float2 mul_w8_3(float2 x) {
  using K = DftConst;
  return float2{rmul(x.y - x.x, K::rh, K::rl), rmul(-x.x - x.y, K::rh, K::rl)};
}

__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = csub_i(t1, t3);
  a3 = cadd_i(t1, t3);
}

__device__ __forceinline__ void dft16(float2 (&v)[16]) {
  using K = DftConst;
#pragma unroll
  for (int b = 0; b < 4; ++b) dft4(v[b], v[b + 4], v[b + 8], v[b + 12]);
  // v[b + 4 k1] holds Y_b[k1]; times W_16^{b k1}.
  v[5] = cmul_const(v[5], K::ch, K::cl, K::sh, K::sl);
  v[9] = mul_w8(v[9]);
  v[13] = cmul_const(v[13], K::sh, K::sl, K::ch, K::cl);
  v[6] = mul_w8(v[6]);
  v[10] = float2{v[10].y, -v[10].x};
  v[14] = mul_w8_3(v[14]);
  v[7] = cmul_const(v[7], K::sh, K::sl, K::ch, K::cl);
  v[11] = mul_w8_3(v[11]);
  v[15] = cmul_const(v[15], -K::ch, -K::cl, -K::sh, -K::sl);
#pragma unroll
  for (int k = 0; k < 4; ++k) dft4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  // v[4 k1 + k2] holds X[k1 + 4 k2]: transpose to natural order (a renaming).
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j) {
      const float2 s = v[4 * i + j];
      v[4 * i + j] = v[4 * j + i];
      v[4 * j + i] = s;
    }
}

// L-point DFT of v[i + S j], j < L, in place (natural order).
template <int L, int S, int V>
__device__ __forceinline__ void dft_strided(float2 (&v)[V], int i) {
  if constexpr (L == 16) {
    dft16(v);
  } else if constexpr (L == 8) {
    float2 e0 = v[i], o0 = v[i + S], e1 = v[i + 2 * S], o1 = v[i + 3 * S];
    float2 e2 = v[i + 4 * S], o2 = v[i + 5 * S], e3 = v[i + 6 * S], o3 = v[i + 7 * S];
    dft4(e0, e1, e2, e3);
    dft4(o0, o1, o2, o3);
    o1 = mul_w8(o1);
    o3 = mul_w8_3(o3);
    v[i] = cadd(e0, o0);
    v[i + 4 * S] = csub(e0, o0);
    v[i + S] = cadd(e1, o1);
    v[i + 5 * S] = csub(e1, o1);
    v[i + 2 * S] = csub_i(e2, o2);
    v[i + 6 * S] = cadd_i(e2, o2);
    v[i + 3 * S] = cadd(e3, o3);
    v[i + 7 * S] = csub(e3, o3);
  } else if constexpr (L == 4) {
    dft4(v[i], v[i + S], v[i + 2 * S], v[i + 3 * S]);
  } else if constexpr (L == 2) {
    const float2 a = v[i], b = v[i + S];
    v[i] = cadd(a, b);
    v[i + S] = csub(a, b);
  }
}

// The last DFTs: V / L of L points, over v[i + (V / L) j].
template <int L, int V>
__device__ __forceinline__ void dft_last(float2 (&v)[V]) {
  if constexpr (L > 1) {
#pragma unroll
    for (int i = 0; i < V / L; ++i) dft_strided<L, V / L>(v, i);
  }
}

// Twiddle W_N^{t k} at entry k * M + t of the table: {re, im} rounded and remainders.
__device__ __forceinline__ float2 tw_mul(float2 v, const float4* tab, int i) {
  const float4 w = tab[i];
  return cmul2f(v, make_float2(w.x, w.y), make_float2(w.z, w.w));
}

template <int V>
__device__ __forceinline__ void conj_all(float2 (&v)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i) v[i].y = -v[i].y;
}

// Slots of the buffer that belong to thread t after a transform (the last exchange's reads).  No
// other thread touches them until the next transform's first exchange, so the thread may keep its
// values there and index them.
template <int N, int V>
struct OwnSlots {
  int base;
  __device__ __forceinline__ explicit OwnSlots(int t)
      : base(N > V * V ? t : t * RegFft<N, V>::Mp) {}
  __device__ __forceinline__ int slot(int m) const { return base + (N > V * V ? m * RegFft<N, V>::M : m); }
};

// Forward transform of the values of thread t; buf[slot * C] is the transform's exchange buffer
// (C interleaved transforms, this one's offset added by the caller), sync() a barrier over the
// threads that share it.  The first sync lets the buffer's earlier contents go.
template <int N, int V, typename Sync>
__device__ __forceinline__ void fft_forward(float2 (&v)[V], int t, float2* buf, int C, const float4* tab, Sync sync) {
  using F = RegFft<N, V>;
  const int q = t % V, u = t / V;
  int wb = t, ws = F::Mp, rb = q * F::Mp + u, rs = F::L, tw = t;
#pragma unroll 1
  for (int pass = 0;; ++pass) {
    dft_strided<V, 1>(v, 0);
    if (N == V * V && pass == 1) return;
#pragma unroll
    for (int k = 1; k < V; ++k) v[k] = tw_mul(v[k], tab, k * F::M + tw);
    sync();
#pragma unroll
    for (int k = 0; k < V; ++k) buf[(wb + k * ws) * C] = v[k];
    sync();
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = buf[(rb + k * rs) * C];
    if (N > V * V && pass == 1) break;
    wb = u * (V * V) + q, ws = V, rb = t, rs = F::M, tw = V * u;
  }
  dft_last<F::L>(v);
}

}  // namespace
}  // namespace pg
