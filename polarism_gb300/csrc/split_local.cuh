// The split-step's local operations at one site (device code shared by the generic column
// pass in split.cu and the register-resident column pass in split_reg.cu): the
// reservoir half steps, the exact nonlinear step and the Wigner increment, for every
// SplitOp.
#pragma once
#include "fft.cuh"
#include "philox.cuh"
#include "pg_internal.h"
#include "split_internal.h"

namespace pg {
namespace {

__device__ __forceinline__ float mul_rn_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn_t(double a, double b) { return __dmul_rn(a, b); }

// psi (1 + dx) (1 + dy) scale, with the factor differences d stored in place of the factors (see
// setup_tables) and scale a power of two; psi is rounded once.  FP32 forms the combined difference first.
// FP64, bound by its arithmetic, adds both small terms to psi together, psi + (t + (psi + t) dy) with
// t = psi dx: 14 instructions instead of 16, and at phases below a radian the combined form's error
// (4.7e-17 rms a kick; two products psi + psi d, as many instructions, round psi twice: 6.7e-17).
__device__ __forceinline__ float2 kick(float2 v, float2 dx, float2 dy, float scale) {
  const float2 dxy = cmul(dx, dy);
  const float2 f1 = make_float2(dx.x + dy.x + dxy.x, dx.y + dy.y + dxy.y);
  const float2 vf = cmul(v, f1);
  return make_float2((v.x + vf.x) * scale, (v.y + vf.y) * scale);
}
__device__ __forceinline__ double2 kick(double2 v, double2 dx, double2 dy, double scale) {
  const double2 t = make_double2(fma(v.x, dx.x, -(v.y * dx.y)), fma(v.x, dx.y, v.y * dx.x));
  const double2 a = make_double2(v.x + t.x, v.y + t.y);
  return make_double2((v.x + fma(a.x, dy.x, fma(-a.y, dy.y, t.x))) * scale,
                      (v.y + fma(a.x, dy.y, fma(a.y, dy.x, t.y))) * scale);
}

// Midpoint RK2 reservoir half step at frozen |psi|^2 with the final clamp
// (polarism/reservoir/single_reservoir.py:100-111).
template <typename T>
__device__ __forceinline__ T reservoir_half(T n, T rho, T pump, T h, const SplitConst<T>& k) {
  const T loss = k.gamma_R + k.R * rho;
  const T k1 = pump - loss * n;
  const T mid = n + T(0.5) * h * k1;
  const T k2 = pump - loss * mid;
  const T out = n + h * k2;
  return out > T(0) ? out : T(0);
}

// Right-hand sides of the two-field reservoirs, state (active, inactive): the double
// reservoir (polarism/reservoir/double_reservoir.py:106-130) and the quadratic-double one,
// fed by kappa n_I^2 (polarism/reservoir/quadratic_double_reservoir.py:13-14).
template <typename T>
__device__ __forceinline__ void two_field_rhs(T a, T b, T rho, T pump, bool quadratic,
                                              const SplitConst<T>& k, T& da, T& db) {
  if (quadratic) {
    const T transfer = k.kappa * b * b;
    da = transfer - k.gamma_R * a - k.R * a * rho;
    db = pump - transfer - k.gamma_I * b;
  } else {
    da = k.R_IA * b - (k.gamma_A + k.R_AI + k.R * rho) * a;
    db = pump - (k.gamma_I + k.R_IA) * b + k.R_AI * a;
  }
}

// The same midpoint half step for both fields of a two-field reservoir, each clamped at 0.
template <typename T>
__device__ __forceinline__ void reservoir_half2(T& a, T& b, T rho, T pump, T h, bool quadratic,
                                                const SplitConst<T>& k) {
  T da, db;
  two_field_rhs(a, b, rho, pump, quadratic, k, da, db);
  T da2, db2;
  two_field_rhs(a + T(0.5) * h * da, b + T(0.5) * h * db, rho, pump, quadratic, k, da2, db2);
  const T na = a + h * da2, nb = b + h * db2;
  a = na > T(0) ? na : T(0);
  b = nb > T(0) ? nb : T(0);
}

// (exp(x) - 1) / x with exp(x) - 1 beside it, and (sin, cos - 1), of the local step: Taylor
// polynomials for |x| < 2^-5 (truncated below 5e-11 relative in FP32, 8e-21 in FP64) and
// |phi| < 1/8 (below 1e-13, 3e-21), the library functions outside.  The per-step arguments are
// that small at the time steps the split-step solvers run with, and the polynomials are cheaper
// than the library's range reduction and division: in FP64, whose two lanes a clock bound the
// pass, about 25 instructions a site instead of some 90.
__device__ __forceinline__ double expm1_over(double x, double* e) {
  if (fabs(x) < 0.03125) {
    double p = fma(x, 1.0 / 362880.0, 1.0 / 40320.0);
    p = fma(x, p, 1.0 / 5040.0);
    p = fma(x, p, 1.0 / 720.0);
    p = fma(x, p, 1.0 / 120.0);
    p = fma(x, p, 1.0 / 24.0);
    p = fma(x, p, 1.0 / 6.0);
    p = fma(x, p, 0.5);
    p = fma(x, p, 1.0);
    *e = x * p;
    return p;
  }
  *e = expm1(x);
  return *e / x;
}
__device__ __forceinline__ float expm1_over(float x, float* e) {
  if (fabsf(x) < 0.03125f) {
    const float p = 1.0f + x * (0.5f + x * (1.0f / 6.0f + x * (1.0f / 24.0f + x * (1.0f / 120.0f))));
    *e = x * p;
    return p;
  }
  *e = expm1f(x);
  return *e / x;
}
__device__ __forceinline__ void local_sincos_m1(double x, double* s, double* cm1) {
  if (fabs(x) < 0.125) {
    const double x2 = x * x;
    double p = fma(x2, -1.0 / 39916800.0, 1.0 / 362880.0);
    p = fma(x2, p, -1.0 / 5040.0);
    p = fma(x2, p, 1.0 / 120.0);
    p = fma(x2, p, -1.0 / 6.0);
    *s = fma(x * x2, p, x);
    double q = fma(x2, 1.0 / 479001600.0, -1.0 / 3628800.0);
    q = fma(x2, q, 1.0 / 40320.0);
    q = fma(x2, q, -1.0 / 720.0);
    q = fma(x2, q, 1.0 / 24.0);
    q = fma(x2, q, -0.5);
    *cm1 = x2 * q;
  } else {
    double c;
    sincos(x, s, &c);
    *cm1 = c - 1.0;
  }
}
__device__ __forceinline__ void local_sincos_m1(float x, float* s, float* cm1) {
  if (fabsf(x) < 0.125f) {
    const float x2 = x * x;
    *s = fmaf(x * x2, fmaf(x2, fmaf(x2, -1.0f / 5040.0f, 1.0f / 120.0f), -1.0f / 6.0f), x);
    *cm1 = x2 * fmaf(x2, fmaf(x2, fmaf(x2, 1.0f / 40320.0f, -1.0f / 720.0f), 1.0f / 24.0f), -0.5f);
  } else {
    float c;
    sincosf(x, s, &c);
    *cm1 = c - 1.0f;  // |phi| >= 1/8: |c - 1| >= 0.0078, so c - 1 keeps c's precision
  }
}

// Exact local step psi * exp(g dt - i phi) (split_step_fft_solver.py:121-139); n2 is the
// inactive reservoir (0 without one), which enters the phase through g_I.  Applied as
// psi + psi D with D = exp(g dt - i phi) - 1 = (e + c1 + e c1) - i (1 + e) s, e = exp(g dt) - 1,
// c1 = cos phi - 1: the factor itself sits next to 1 at these step sizes, where its rounding
// would repeat step after step (a rounded exp(g dt) there carries up to 6e-8 of bias a step).
template <typename T>
__device__ __forceinline__ void nonlinear(T& re, T& im, T n, T n2, bool two, T vre, T vim, T dt,
                                          const SplitConst<T>& k) {
  const T rho = re * re + im * im;
  const T gain = (k.R * n - k.gamma_C) * T(0.5) + vim * k.inv_hbar;
  // (exp(2 y) - 1) / (2 y) = p (1 + e / 2) with y = gain dt, e = exp(y) - 1, p = e / y
  T e;
  const T p = expm1_over(gain * dt, &e);
  const T phase_time = dt * (p + p * (T(0.5) * e));
  T pot = vre + k.g_R * n;
  if (two) pot += k.g_I * n2;
  const T phase = (pot * dt + k.g_C * rho * phase_time) * k.inv_hbar;
  T s, c1;
  local_sincos_m1(phase, &s, &c1);
  const T dre = e + c1 + e * c1;
  const T dim = -(s + e * s);
  const T r = re, i = im;
  re = r + (r * dre - i * dim);
  im = i + (r * dim + i * dre);
}


// Everything the local step of one column-pass launch needs for a member, and the step at
// one site (flat index o within the member's plane).
template <typename T>
struct LocalStep {
  using C2 = typename C2T<T>::type;
  SplitConst<T> k;
  // The launch's settings, copied (a pointer to the kernel's parameter would move it to local
  // memory and make every read a local load).
  int op, reservoir, noise, pot_kind;
  long long pump_term_stride;
  int m_count, L;
  const T* c0;
  const T* c1;
  T s0, s1;
  const T* pm;
  const T* vm;
  T* rm;
  T* rm2;
  bool two, quadratic;
  T dt, h;
  PhiloxCellPrefix prefix;

  __device__ __forceinline__ LocalStep(const ColPassArgs& args, int member, T* res, const T* pump,
                                       const T* potential, const SplitConst<T>* consts,
                                       const T* scales, const unsigned long long* step_base) {
    op = args.op;
    reservoir = args.reservoir;
    noise = args.noise;
    pot_kind = args.potential;
    pump_term_stride = args.pump_term_stride;
    k = consts[member];
    m_count = args.members;
    // Coefficients [k][sample][term][member]; the term axis exists only with several lasers.
    L = args.pump_terms > 1 ? args.pump_terms : 1;
    c0 = scales + static_cast<long long>((args.scale_offset + 0) * L) * m_count + member;
    c1 = scales + static_cast<long long>((args.scale_offset + 1) * L) * m_count + member;
    s0 = c0[0];
    s1 = c1[0];
    const long long plane = static_cast<long long>(args.nx) * args.ny;
    pm = pump + member * args.pump_stride;
    vm = potential ? potential + member * args.pot_stride * (args.potential == 2 ? 2 : 1) : nullptr;
    rm = res + member * plane;
    // Second reservoir field (inactive) one field after the first: [field][member][y][x].
    two = args.res_kind >= 2;
    quadratic = args.res_kind == 3;
    rm2 = two ? rm + static_cast<long long>(args.members) * plane : nullptr;
    dt = args.template dt_of<T>();
    h = dt * T(0.5);
    const unsigned long long step = args.noise ? step_base[0] + args.step_offset : 0ull;
    // Philox rounds that depend only on (step, stream, key), formed once per launch and member.
    prefix = philox_cell_prefix(static_cast<uint32_t>(step), static_cast<uint32_t>(step >> 32), 1u,
                                static_cast<uint32_t>(k.seed), static_cast<uint32_t>(k.seed >> 32));
  }

  // One reservoir half step at the given pump value on the chosen reservoir model.
  __device__ __forceinline__ void res_half(T& n, T& n2, T rho, T pump_value) const {
    if (two) {
      reservoir_half2(n, n2, rho, pump_value, h, quadratic, k);
    } else if (reservoir) {
      n = reservoir_half(n, rho, pump_value, h, k);
    }
  }

  // Whether step_single covers this launch: one reservoir field, one laser and no potential
  // (the common case, without the general code's branches).
  __device__ __forceinline__ bool single() const {
    return reservoir && !two && L == 1 && vm == nullptr;
  }

  // apply() for that case with the operation known at compile time, on values already
  // loaded: the reservoir n and the envelope P at site o (32-bit site offsets: a member holds
  // fewer than 2^31 sites).  The same operations, in the same order; returns the new n, which
  // the caller stores unless OP is SPLIT_OP_NONLINEAR.
  template <int OP, bool NOISE>
  __device__ __forceinline__ T step_single(C2& v, T n, T P, int o) const {
    if (OP == SPLIT_OP_KOUTER) {
      n = reservoir_half(n, v.x * v.x + v.y * v.y, mul_rn_t(s0, P), h, k);
      nonlinear(v.x, v.y, n, T(0), false, T(0), T(0), dt, k);
      n = reservoir_half(n, v.x * v.x + v.y * v.y, mul_rn_t(s1, P), h, k);
    } else if (OP == SPLIT_OP_RES_START || OP == SPLIT_OP_RES_END) {
      n = reservoir_half(n, v.x * v.x + v.y * v.y, mul_rn_t(s0, P), h, k);
    } else if (OP == SPLIT_OP_RES_END_START) {
      const T rho = v.x * v.x + v.y * v.y;
      n = reservoir_half(n, rho, mul_rn_t(s0, P), h, k);
      n = reservoir_half(n, rho, mul_rn_t(s1, P), h, k);
    } else if (OP == SPLIT_OP_NONLINEAR) {
      nonlinear(v.x, v.y, n, T(0), false, T(0), T(0), dt, k);
    }
    if (NOISE && (OP == SPLIT_OP_KOUTER || OP == SPLIT_OP_NONLINEAR)) {
      const uint32_t cell[1] = {static_cast<uint32_t>(o)};
      Words4 w[1];
      philox_cells(cell, prefix, w);
      WignerDraw<T>::apply(w[0], k.noise_a + k.noise_b * n, v.x, v.y);
    }
    return n;
  }

  // What the step reads at a site of any launch: the reservoir fields, the pump at the first and
  // the second coefficient sample, the potential.
  struct Inputs {
    T n, n2, Pa, Pb, vre, vim;
  };
  __device__ __forceinline__ Inputs load(long long o) const {
    Inputs s;
    s.n = (reservoir || two) ? rm[o] : T(0);
    s.n2 = two ? rm2[o] : T(0);
    if (L > 1) {
      s.Pa = pump_terms_value(pm, pump_term_stride, c0, m_count, L, o);
      s.Pb = pump_terms_value(pm, pump_term_stride, c1, m_count, L, o);
    } else {
      const T P = pm[o];
      s.Pa = mul_rn_t(s0, P);
      s.Pb = mul_rn_t(s1, P);
    }
    s.vre = s.vim = T(0);
    if (vm) {
      s.vre = pot_kind == 2 ? vm[2 * o] : vm[o];
      s.vim = pot_kind == 2 ? vm[2 * o + 1] : T(0);
    }
    return s;
  }
  // The step on those values: v and the reservoir fields of s advance.
  template <int OP, bool NOISE>
  __device__ __forceinline__ void compute(C2& v, Inputs& s, long long o) const {
    const T rho = v.x * v.x + v.y * v.y;
    if (OP == SPLIT_OP_KOUTER) {
      res_half(s.n, s.n2, rho, s.Pa);
      nonlinear(v.x, v.y, s.n, s.n2, two, s.vre, s.vim, dt, k);
      res_half(s.n, s.n2, v.x * v.x + v.y * v.y, s.Pb);
    } else if (OP == SPLIT_OP_RES_START || OP == SPLIT_OP_RES_END) {
      res_half(s.n, s.n2, rho, s.Pa);
    } else if (OP == SPLIT_OP_RES_END_START) {
      res_half(s.n, s.n2, rho, s.Pa);
      res_half(s.n, s.n2, rho, s.Pb);
    } else if (OP == SPLIT_OP_NONLINEAR) {
      nonlinear(v.x, v.y, s.n, s.n2, two, s.vre, s.vim, dt, k);
    }
    if (NOISE && (OP == SPLIT_OP_KOUTER || OP == SPLIT_OP_NONLINEAR)) {
      const uint32_t cell[1] = {static_cast<uint32_t>(o)};
      Words4 w[1];
      philox_cells(cell, prefix, w);
      WignerDraw<T>::apply(w[0], k.noise_a + k.noise_b * s.n, v.x, v.y);
    }
  }
  __device__ __forceinline__ void store(const Inputs& s, long long o) const {
    if (reservoir || two) rm[o] = s.n;
    if (two) rm2[o] = s.n2;
  }
  __device__ __forceinline__ void apply(C2& v, long long o) const {
    Inputs s = load(o);
    switch (op * 2 + (noise ? 1 : 0)) {
#define PG_SPLIT_OP(OP)                      \
  case OP * 2: compute<OP, false>(v, s, o); break; \
  case OP * 2 + 1: compute<OP, true>(v, s, o); break;
      PG_SPLIT_OP(SPLIT_OP_KOUTER)
      PG_SPLIT_OP(SPLIT_OP_NONLINEAR)
      PG_SPLIT_OP(SPLIT_OP_RES_START)
      PG_SPLIT_OP(SPLIT_OP_RES_END)
      PG_SPLIT_OP(SPLIT_OP_RES_END_START)
#undef PG_SPLIT_OP
      default:
        break;
    }
    store(s, o);
  }
};

}  // namespace
}  // namespace pg
