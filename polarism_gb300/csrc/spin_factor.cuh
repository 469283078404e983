// The two-component Lawson factor of one mode in FP32 (device code of the IFRK row passes): out =
// sum_t coef_t / N exp(-i H(k) tau_t / hbar) src_t with exp(-i H t) = exp(-i E t) [[cos - i s z,
// -i s u], [-i s u*, cos + i s z]], s = sin(w t) / w, w = sqrt(z^2 + |u|^2), u = beta (kx - i ky)^2
// (polarism/dispersion.py:66-83).
#pragma once
#include "ifrk_internal.h"

namespace pg {
namespace {

// sin and cos of (r_hi + r_lo)(t_hi + t_lo): the product is formed as p + t with the exact
// rounding error of p = r_hi t_hi (an FMA) and the cross terms, reduced by 2 pi split into two
// floats (Cody and Waite's method), so the reduced angle carries an absolute error of a few
// 1e-7 for any angle below 2^24 turns -- the accuracy of the FP64 reduction rounded to FP32.
__device__ __forceinline__ void sincos_product(float r_hi, float r_lo, float t_hi, float t_lo,
                                               float* s, float* c) {
  constexpr float kTwoPiHi = 6.28318548202514648f;        // float(2 pi)
  constexpr float kTwoPiLo = -1.74845553146951617e-07f;   // 2 pi - kTwoPiHi
  constexpr float kInvTwoPi = 0.159154943091895336f;
  const float p = r_hi * t_hi;
  const float e = fmaf(r_hi, t_hi, -p);
  const float t = fmaf(r_hi, t_lo, fmaf(r_lo, t_hi, e));
  const float n = rintf(p * kInvTwoPi);
  const float d = fmaf(-n, kTwoPiLo, fmaf(-n, kTwoPiHi, p)) + t;
  sincosf(d, s, c);
}

// One mode's row of the FP32 table (spin_mode_table_kernel).
struct SpinMode {
  float re_hi, re_lo, rw_hi, rw_lo, ure, uim, inv_om;
};
__device__ __forceinline__ SpinMode load_spin_mode(const float* tm, long long plane) {
  return SpinMode{tm[0],         tm[plane],     tm[2 * plane], tm[3 * plane],
                  tm[4 * plane], tm[5 * plane], tm[6 * plane]};
}

// acc += w exp(-i H tau / hbar) (s0, s1).
__device__ __forceinline__ void spin_term(const SpinMode& q, float tau_hi, float tau_lo, float w, float zf,
                                          float inv_hbar, float2 s0, float2 s1, float2& acc0,
                                          float2& acc1) {
  float se, ce, sw, cw;
  sincos_product(q.re_hi, q.re_lo, tau_hi, tau_lo, &se, &ce);
  sincos_product(q.rw_hi, q.rw_lo, tau_hi, tau_lo, &sw, &cw);
  const float so = q.inv_om > 0.0f ? sw * q.inv_om : tau_hi * inv_hbar;
  const float sz = so * zf;
  const float2 a0{cw * s0.x + sz * s0.y + so * (q.uim * s1.x + q.ure * s1.y),
                  cw * s0.y - sz * s0.x + so * (q.uim * s1.y - q.ure * s1.x)};
  const float2 a1{cw * s1.x - sz * s1.y + so * (q.ure * s0.y - q.uim * s0.x),
                  cw * s1.y + sz * s1.x - so * (q.ure * s0.x + q.uim * s0.y)};
  // phase exp(-i E t) = (ce, -se)
  acc0.x += w * (ce * a0.x + se * a0.y);
  acc0.y += w * (ce * a0.y - se * a0.x);
  acc1.x += w * (ce * a1.x + se * a1.y);
  acc1.y += w * (ce * a1.y - se * a1.x);
}

}  // namespace
}  // namespace pg
