// The site step of the IFRK column passes for the common configuration (device code shared by
// the generic column pass in ifrk.cu and the 1024-point register-resident column pass in
// ifrk_col_fast.cu): one field component, one single reservoir, one laser.  Math as
// polarism/solver/ifrk_fft_cuda_solver.py:128-142 (right-hand side) and :148-241 (stage
// reservoir n0 + sum_j coef_j dn_j, single-reservoir derivative, step-end clamp and Wigner
// increment), restated from the generic loop of ifrk_col_kernel, which covers every other
// configuration.
#pragma once
#include "fft.cuh"
#include "ifrk_internal.h"
#include "philox.cuh"
#include "pg_internal.h"

namespace pg {
namespace {

__device__ __forceinline__ float mul_rn_i(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn_i(double a, double b) { return __dmul_rn(a, b); }

// Whether the column pass's site step has the batched form: one component, one single
// reservoir, one laser, a stage (mode 0, up to five terms) or the step end (mode 1, one to five
// terms).  Lawson RK4 and Dormand-Prince 5 have at most five nonzero terms in a tableau row.
__host__ __device__ inline bool ifrk_sites_batched(const IfrkColArgs& a) {
  const bool base = a.comps == 1 && a.res_fields == 1 && a.res_comps == 1 && a.pump_terms <= 1;
  return base && ((a.mode == 0 && a.terms <= 5) || (a.mode == 1 && a.terms >= 1 && a.terms <= 5));
}

// The sites a thread works on, of a panel of C = 2^lc columns of ny rows held as [row][column] and dealt
// over the block: site e = first, first + step, ... below count, at element o of the member's plane and
// element `slot` of the panel.
struct PanelSites {
  int C, lc, nx, x0, total;
  __device__ __forceinline__ int first() const { return static_cast<int>(threadIdx.x); }
  __device__ __forceinline__ int step() const { return static_cast<int>(blockDim.x); }
  __device__ __forceinline__ int count() const { return total; }
  __device__ __forceinline__ void at(int e, int& slot, int& o) const {
    const int c = e & (C - 1), i = e >> lc;
    o = i * nx + x0 + c;
    slot = i * C + c;
  }
};

// A stage (MODE 0) or step end (MODE 1) over a thread's sites (the member's plane at mbase).
// Each thread takes U sites at a time and issues every global load of the batch (reservoir, the TERMS stage
// derivatives, envelope, potential) before it forms the first result, so U sites' loads are
// in flight; one site at a time, a site's stores would come before the next site's loads,
// which the compiler may not move above them.  The arithmetic is the generic loop's,
// expression for expression and in the same order.
template <typename T, int MODE, int TERMS, int U>
__device__ __forceinline__ void ifrk_sites_single(
    typename C2T<T>::type* buf, const PanelSites& sites, const IfrkColArgs& a,
    const SplitConst<T>& k, long long mbase, const T* __restrict__ n0,
    T* __restrict__ dn_out, T* __restrict__ n_out, typename C2T<T>::type* __restrict__ psi_start,
    typename C2T<T>::type* __restrict__ psi_new, const T* __restrict__ pm,
    const T* __restrict__ vm, T s0, const PhiloxCellPrefix& prefix) {
  using C2 = typename C2T<T>::type;
  const int count = sites.count();
  const T* dn[TERMS > 0 ? TERMS : 1];
  T cf[TERMS > 0 ? TERMS : 1];
#pragma unroll
  for (int j = 0; j < TERMS; ++j) {
    dn[j] = static_cast<const T*>(a.dn[j]) + mbase;
    cf[j] = static_cast<T>(a.coef[j]);
  }
  const T* nm = n0 + mbase;
  const int step = sites.step();
#pragma unroll 1
  for (int e0 = sites.first(); e0 < count; e0 += U * step) {
    int o[U], bi[U];
    bool ok[U];
    C2 v[U];
    T nv[U], acc[U], pp[U], vre[U], vim[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * step;
      ok[u] = e < count;
      sites.at(ok[u] ? e : e0, bi[u], o[u]);  // e0: loads stay in bounds
      v[u] = buf[bi[u]];
      nv[u] = nm[o[u]];
      acc[u] = T(0);
      if (MODE == 0) {
        pp[u] = pm[o[u]];
        vre[u] = T(0);
        vim[u] = T(0);
        if (vm) {
          vre[u] = a.potential == 2 ? vm[2 * static_cast<long long>(o[u])] : vm[o[u]];
          vim[u] = a.potential == 2 ? vm[2 * static_cast<long long>(o[u]) + 1] : T(0);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < TERMS; ++j)
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u] += cf[j] * dn[j][o[u]];
    if (MODE == 0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        const T nval = nv[u] + acc[u];
        const C2 x = v[u];
        const T rho = x.x * x.x + x.y * x.y;
        if (psi_start) psi_start[mbase + o[u]] = x;
        const T eff = vre[u] + k.g_C * rho + k.g_R * nval;
        const T e_over = eff * k.inv_hbar;
        const T g = T(0.5) * (k.R * nval - k.gamma_C) + vim[u] * k.inv_hbar;
        buf[bi[u]] = C2{g * x.x + e_over * x.y, g * x.y - e_over * x.x};
        const T P = mul_rn_i(s0, pp[u]);
        dn_out[mbase + o[u]] = P - (k.gamma_R + k.R * rho) * nval;
      }
    } else {
      Words4 w[U];
      if (a.noise) {
        uint32_t cell[U];
#pragma unroll
        for (int u = 0; u < U; ++u) cell[u] = static_cast<uint32_t>(o[u]);
        philox_cells(cell, prefix, w);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        T nval = nv[u] + acc[u];
        nval = nval > T(0) ? nval : T(0);
        n_out[mbase + o[u]] = nval;
        C2 x = v[u];
        if (a.noise) {
          WignerDraw<T>::apply(w[u], k.noise_a + k.noise_b * nval, x.x, x.y);
          buf[bi[u]] = x;
        }
        psi_new[mbase + o[u]] = x;
      }
    }
  }
}

// ifrk_sites_single for the launch's mode and term count (ifrk_sites_batched(a) holds); U0 /
// U1 sites a batch at a stage / the step end.
template <typename T, int U0, int U1>
__device__ __forceinline__ void ifrk_sites_run(
    typename C2T<T>::type* buf, const PanelSites& sites, const IfrkColArgs& a,
    const SplitConst<T>& k, long long mbase, const T* n0, T* dn_out, T* n_out,
    typename C2T<T>::type* psi_start, typename C2T<T>::type* psi_new, const T* pm, const T* vm,
    T s0, const PhiloxCellPrefix& prefix) {
  switch (a.mode * 8 + a.terms) {
#define PG_IFRK_SITES(MODE, TERMS, U)                                                         \
  case MODE * 8 + TERMS:                                                                      \
    ifrk_sites_single<T, MODE, TERMS, U>(buf, sites, a, k, mbase, n0, dn_out, n_out, \
                                         psi_start, psi_new, pm, vm, s0, prefix);             \
    break;
    PG_IFRK_SITES(0, 0, U0)
    PG_IFRK_SITES(0, 1, U0)
    PG_IFRK_SITES(0, 2, U0)
    PG_IFRK_SITES(0, 3, U0)
    PG_IFRK_SITES(0, 4, U0)
    PG_IFRK_SITES(0, 5, U0)
    PG_IFRK_SITES(1, 1, U1)
    PG_IFRK_SITES(1, 2, U1)
    PG_IFRK_SITES(1, 3, U1)
    PG_IFRK_SITES(1, 4, U1)
    PG_IFRK_SITES(1, 5, U1)
#undef PG_IFRK_SITES
    default:
      break;
  }
}

template <typename T>
__device__ __forceinline__ T scaled_square(T mag, T scale) {
  // (mag / scale)^2 with the reference's handling of a zero scale.
  if (scale > T(0)) {
    const T r = mag / scale;
    return r * r;
  }
  return mag == T(0) ? T(0) : T(INFINITY);
}

// The site step of every configuration on values already loaded: v the field components (a stage
// replaces them by the right-hand side, a noisy step end adds the Wigner increment), nval the
// stage or final reservoir values and dsum their increments at elements ridx, o the site in the
// plane.
template <typename T>
struct IfrkGeneral {
  using C2 = typename C2T<T>::type;
  const IfrkColArgs& a;
  const SplitConst<T>& k;
  T s0;
  const T* cs;
  const T* pm;
  const T* vm;
  const T* n0;
  T* dn_out;
  T* n_out;
  C2* psi_start;
  C2* psi_new;
  long long fbase, plane;
  const PhiloxCellPrefix (&prefix)[2];

  // The stage's envelope and potential at site o: loaded with the reservoirs, before any store.
  struct Site {
    T pump, vre, vim;
  };
  __device__ __forceinline__ Site load(long long o) const {
    Site p{T(0), T(0), T(0)};
    if (a.mode != 0) return p;
    if (a.res_fields >= 1 && !(a.pump_terms > 1 && cs)) p.pump = pm[o];
    if (vm) {
      p.vre = a.potential == 2 ? vm[2 * o] : vm[o];
      p.vim = a.potential == 2 ? vm[2 * o + 1] : T(0);
    }
    return p;
  }

  __device__ __forceinline__ void apply(C2 (&v)[2], T (&nval)[4], const T (&dsum)[4], const Site& site,
                                        const long long (&ridx)[4], long long o, double& local) const {
    const int comps = a.comps, F = a.res_fields, Cr = a.res_comps, NQ = F * Cr;
    const int L = a.pump_terms > 1 ? a.pump_terms : 1;
    if (a.mode == 0) {
      T rho[2];
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        rho[comp] = v[comp].x * v[comp].x + v[comp].y * v[comp].y;
        if (comp < comps && psi_start) psi_start[fbase + comp * plane + o] = v[comp];
      }
      C2 out[2];
      const T vre = site.vre, vim = site.vim;
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        if (comp >= comps) break;
        const int ra = Cr == comps ? comp : 0;
        const T nA = F >= 1 ? nval[ra] : T(0);
        const T nI = F == 2 ? nval[Cr + ra] : T(0);
        // rhs = (-i/hbar) (V_re + g_C rho + alpha_2 rho_other + g_R n_A + g_I n_I) psi
        //       + (R n_A - gamma_C)/2 psi + (V_im / hbar) psi
        T eff = vre + k.g_C * rho[comp] + k.g_R * nA;
        if (comps == 2) eff += k.alpha_2 * rho[1 - comp];
        if (F == 2) eff += k.g_I * nI;
        const T e_over = eff * k.inv_hbar;
        const T g = T(0.5) * (k.R * nA - k.gamma_C) + vim * k.inv_hbar;
        out[comp] = C2{g * v[comp].x + e_over * v[comp].y, g * v[comp].y - e_over * v[comp].x};
      }
#pragma unroll
      for (int comp = 0; comp < 2; ++comp)
        if (comp < comps) v[comp] = out[comp];
      if (F >= 1) {
        const T p_site = L > 1 && cs ? pump_terms_value(pm, a.pump_term_stride, cs, a.members, L, o)
                                     : mul_rn_i(s0, site.pump);
#pragma unroll
        for (int cr = 0; cr < 2; ++cr) {
          if (cr >= Cr) break;
          const T rr = Cr == comps ? rho[cr] : (comps == 2 ? rho[0] + rho[1] : rho[0]);
          const T P = Cr == 2 ? mul_rn_i(p_site, k.weight[cr]) : p_site;
          if (F == 1) {
            dn_out[ridx[cr]] = P - (k.gamma_R + k.R * rr) * nval[cr];
          } else if (a.res_kind == PG_RES_QDOUBLE) {
            // quadratic_double_reservoir.py:13-14: n_R fed by kappa n_I^2.
            const T nR = nval[cr], nI = nval[Cr + cr];
            const T transfer = k.kappa * nI * nI;
            dn_out[ridx[cr]] = transfer - k.gamma_R * nR - k.R * nR * rr;
            dn_out[ridx[Cr + cr]] = P - transfer - k.gamma_I * nI;
          } else {
            const T nA = nval[cr], nI = nval[Cr + cr];
            dn_out[ridx[Cr + cr]] = P - (k.gamma_I + k.R_IA) * nI + k.R_AI * nA;
            dn_out[ridx[cr]] = k.R_IA * nI - (k.gamma_A + k.R_AI + k.R * rr) * nA;
          }
        }
      }
    } else if (a.mode == 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= NQ) break;
        nval[q] = nval[q] > T(0) ? nval[q] : T(0);
        n_out[ridx[q]] = nval[q];
      }
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        if (comp >= comps) break;
        C2 w = v[comp];
        if (a.noise) {
          const T nA = F >= 1 ? nval[Cr == comps ? comp : 0] : T(0);
          const uint32_t cell[1] = {static_cast<uint32_t>(o)};
          Words4 w1[1];
          philox_cells(cell, prefix[comp], w1);
          const Words4 words = w1[0];
          WignerDraw<T>::apply(words, k.noise_a + k.noise_b * nA, w.x, w.y);
          v[comp] = w;
        }
        psi_new[fbase + comp * plane + o] = w;
      }
    } else {  // mode 2: error norm, v = condensate error, dsum = reservoir error
#pragma unroll
      for (int comp = 0; comp < 2; ++comp) {
        if (comp >= comps) break;
        const C2 y0 = psi_start[fbase + comp * plane + o];
        const C2 y1 = psi_new[fbase + comp * plane + o];
        const T a0 = sqrt(y0.x * y0.x + y0.y * y0.y), a1 = sqrt(y1.x * y1.x + y1.y * y1.y);
        const T scale = static_cast<T>(a.atol) + static_cast<T>(a.rtol) * (a0 > a1 ? a0 : a1);
        local += static_cast<double>(
            scaled_square(sqrt(v[comp].x * v[comp].x + v[comp].y * v[comp].y), scale));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= NQ) break;
        const T r0 = fabs(n0[ridx[q]]), r1 = fabs(n_out[ridx[q]]);
        const T rs = static_cast<T>(a.atol) + static_cast<T>(a.rtol) * (r0 > r1 ? r0 : r1);
        local += static_cast<double>(scaled_square(fabs(dsum[q]), rs));
      }
    }
  }
};

}  // namespace
}  // namespace pg
