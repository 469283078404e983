// The finite-difference right-hand side at one site in either precision, with every option of
// the general kernels: potential, kinetic relaxation, no / single / two-field reservoirs.
//
// Math follows polarism/model.py:89-127, polarism/reservoir/single_reservoir.py:81-98,
// double_reservoir.py:106-130 (n_I feeding n_A) and quadratic_double_reservoir.py:13-14 (n_I
// feeding n_R through kappa n_I^2).  Every operation and its fused multiply-add is spelled out in
// the order of rk4_site.cuh, so that the streaming kernel (rk4.cu), the tile kernel
// (rk4_tile.cuh) and the full-width kernels give the same bits for the same site.
#pragma once
#include <cuda_runtime.h>

#include "pg_internal.h"

namespace pg {
namespace {

template <typename T>
struct Cplx;
template <>
struct Cplx<float> {
  using type = float2;
};
template <>
struct Cplx<double> {
  using type = double2;
};

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// One evaluation.  c is the centre, (lt, rt, up, dn) the four neighbours, n the active
// reservoir density, n2 the inactive one, sP the scaled pump, (vre, vim) the potential; writes
// d = dpsi/dt, dnr = dn/dt and dn2 = dn2/dt.
template <typename T, bool GENERAL, bool TWO>
__device__ __forceinline__ void general_rhs(const typename Cplx<T>::type c,
                                            const typename Cplx<T>::type lt,
                                            const typename Cplx<T>::type rt,
                                            const typename Cplx<T>::type up,
                                            const typename Cplx<T>::type dn, const T n, const T sP,
                                            const RhsConst<T>& k, const T vre, const T vim,
                                            const RK4Features& f, typename Cplx<T>::type& d, T& dnr,
                                            const T n2, T& dn2) {
  // -a (Laplacian without its centre weight)
  const T nlx = fma_t(-k.ay, pump_add_rn(up.x, dn.x), pump_mul_rn(-k.ax, pump_add_rn(lt.x, rt.x)));
  const T nly = fma_t(-k.ay, pump_add_rn(up.y, dn.y), pump_mul_rn(-k.ax, pump_add_rn(lt.y, rt.y)));
  const T rho = fma_t(c.x, c.x, pump_mul_rn(c.y, c.y));
  T w = fma_t(k.gr, n, fma_t(k.gc, rho, k.w0));
  T gl = fma_t(k.half_R, n, -k.half_gC);
  if (GENERAL) {
    w = fma_t(vre, k.inv_hbar, w);
    gl = fma_t(vim, k.inv_hbar, gl);
    if (TWO) w = fma_t(k.gi, n2, w);
  }
  const T ux = fma_t(w, c.x, nlx), uy = fma_t(w, c.y, nly);  // w c - a lap_neighbours
  d.x = fma_t(gl, c.x, uy);
  d.y = fma_t(gl, c.y, -ux);
  if (GENERAL && f.relax) {
    const T en = pump_mul_rn(k.eta_a, n);  // the Laplacian with its centre weight is -(w0 c + nl)
    d.x = fma_t(-en, fma_t(k.w0, c.x, nlx), d.x);
    d.y = fma_t(-en, fma_t(k.w0, c.y, nly), d.y);
  }
  dnr = fma_t(-fma_t(k.R, rho, k.gamma_R), n, sP);
  dn2 = T(0);
  if (GENERAL) {
    if (f.reservoir == 0) {
      dnr = T(0);
    } else if (TWO && f.reservoir == 2) {
      dn2 = fma_t(k.R_AI, n, fma_t(-pump_add_rn(k.gamma_I, k.R_IA), n2, sP));
      dnr = fma_t(-fma_t(k.R, rho, pump_add_rn(k.gamma_A, k.R_AI)), n, pump_mul_rn(k.R_IA, n2));
    } else if (TWO && f.reservoir == 3) {
      const T transfer = pump_mul_rn(pump_mul_rn(k.kappa, n2), n2);
      dnr = fma_t(-fma_t(k.R, rho, k.gamma_R), n, transfer);
      dn2 = fma_t(-k.gamma_I, n2, pump_add_rn(sP, -transfer));
    }
  }
}

// y + h d
template <typename T>
__device__ __forceinline__ typename Cplx<T>::type axpy_t(T h, typename Cplx<T>::type d,
                                                         typename Cplx<T>::type y) {
  return typename Cplx<T>::type{fma_t(h, d.x, y.x), fma_t(h, d.y, y.y)};
}

}  // namespace
}  // namespace pg
