// FP32 Lawson IFRK passes on the register-resident transforms (fft_reg.cuh): rows and columns of
// 64 to 4096 points, one component or the two-component spinor.  The passes and their arithmetic
// per site and mode are those of ifrk.cu.
//
// Two components: the threads of a row (or panel) hold one component each.  The steps that couple
// the components -- the Lawson factor of a mode, the site step -- run with the values parked in
// each thread's own slots of the exchange buffer: of the V sites or modes that a pair of threads
// holds (same position, one component each), the first thread takes the first half and the second
// the other half, both components of each.
#include "ifrk_internal.h"
#include "ifrk_sites.cuh"
#include "reg_pass.cuh"
#include "spin_factor.cuh"

namespace pg {
namespace {

// Two components are bound by the latency of the coupled steps, not by registers or warps: a thread
// takes kPairModes modes through the Lawson terms together (their loads and sines independent of one
// another) with 128 registers, and the column pass may use twice the registers where more than one
// block would fit.  A Dormand-Prince trial: 64^2 263 -> 226 us, 256^2 299 -> 260 us, 512^2 432 -> 415 us,
// 2048^2 4.86 -> 4.66 ms.  Two modes are 2 % slower, one with the next one's loads ahead 6 %; two sites
// at a time in the column pass spill (512^2 474 us).
constexpr int kPairModes = 4;

template <int N, int V, int COMPS>
__global__ void __launch_bounds__(RowShape<N, V, COMPS>::MAX_THREADS,
                                  (COMPS == 2 ? 512 : 1024) / RowShape<N, V, COMPS>::MAX_THREADS)
    ifrk_row_reg_kernel(const float2* __restrict__ in, float2* __restrict__ save,
                        float2* __restrict__ out, const float2* __restrict__ tables,
                        const float4* __restrict__ tab, const __grid_constant__ IfrkRowArgs a) {
  using S = RowShape<N, V, COMPS>;
  constexpr int M = S::M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int t = threadIdx.x % M, group = threadIdx.x / M;  // group: (row, component)
  const int comp = COMPS == 2 ? group & 1 : 0, r = group / COMPS;
  const int member = blockIdx.z;
  const int row = blockIdx.x * a.rows + r;
  float2* buf = reinterpret_cast<float2*>(smem_raw) + group * S::STRIDE;
  const GroupSync<(M <= 32)> sync{1 + group, M};
  const GroupSync<(M * COMPS <= 32)> pair_sync{8 + r, M * COMPS};
  const long long plane = static_cast<long long>(N) * a.ny;
  const long long moff = member * a.member_stride + static_cast<long long>(row) * N;
  const long long own = moff + comp * plane + t;
  float2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = in ? in[own + m * M] : make_float2(0.f, 0.f);
  // Phase 0: forward transform, save, combination; phase 1: the inverse transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.forward : a.inverse) {
      if (ph == 1) conj_all(v);
      fft_forward<N, V>(v, t, buf, 1, tab, sync);
      if (ph == 1) conj_all(v);
    }
    if (ph == 1) continue;
    if (save) {
#pragma unroll
      for (int m = 0; m < V; ++m) save[own + m * M] = v[m];
    }
    if constexpr (COMPS == 1) {
      // The term on this row's own spectrum (src null; at most one) first, in place, then the
      // stored spectra, a term at a time so that the row stays the only array in registers.
      const long long table_stride = static_cast<long long>(a.members) * (N + a.ny);
      const float2* tabs = tables + static_cast<long long>(member) * (N + a.ny);
      int self = -1;
      for (int s = 0; s < a.terms; ++s)
        if (a.src[s] == nullptr) self = s;
      if (self >= 0) {
        const float2* e = tabs + a.table[self] * table_stride;
        const float2 ey = e[N + row];
        const float c = static_cast<float>(a.coef[self]);
#pragma unroll
        for (int m = 0; m < V; ++m) {
          const float2 ev = cmul(cmul(e[t + m * M], ey), v[m]);
          v[m] = make_float2(c * ev.x, c * ev.y);
        }
      } else {
#pragma unroll
        for (int m = 0; m < V; ++m) v[m] = make_float2(0.f, 0.f);
      }
#pragma unroll 1
      for (int s = 0; s < a.terms; ++s) {
        if (s == self) continue;
        const float2* e = tabs + a.table[s] * table_stride;
        const float2* src = static_cast<const float2*>(a.src[s]) + own;
        const float2 ey = e[N + row];
        const float c = static_cast<float>(a.coef[s]);
#pragma unroll
        for (int m = 0; m < V; ++m) {
          const float2 ev = cmul(cmul(e[t + m * M], ey), src[m * M]);
          v[m].x += c * ev.x;
          v[m].y += c * ev.y;
        }
      }
    } else {
      constexpr int U = kPairModes;
      const OwnSlots<N, V> slots(t);
#pragma unroll
      for (int m = 0; m < V; ++m) buf[slots.slot(m)] = v[m];
      pair_sync();
      float2* b0 = buf - comp * S::STRIDE;
      float2* b1 = b0 + S::STRIDE;
      const SpinorConst sc = static_cast<const SpinorConst*>(a.spin)[member];
      const float zf = static_cast<float>(sc.half_z), inv_hbar = static_cast<float>(sc.inv_hbar);
      const float* modes = a.modes + static_cast<long long>(member) * kSpinModeFields * plane +
                           static_cast<long long>(row) * N + t;
#pragma unroll 1
      for (int h = 0; h < V / 2; h += U) {
        SpinMode mode[U];
        float2 self0[U], self1[U], acc0[U], acc1[U];
        const int m0 = comp * (V / 2) + h;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          mode[u] = load_spin_mode(modes + (m0 + u) * M, plane);
          const int slot = slots.slot(m0 + u);
          self0[u] = b0[slot];
          self1[u] = b1[slot];
          acc0[u] = acc1[u] = make_float2(0.f, 0.f);
        }
#pragma unroll 1
        for (int s = 0; s < a.terms; ++s) {
          float2 s0[U], s1[U];
          const float2* src = static_cast<const float2*>(a.src[s]);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            s0[u] = self0[u];
            s1[u] = self1[u];
            if (src) {
              const long long at = moff + t + (m0 + u) * M;
              s0[u] = src[at];
              s1[u] = src[at + plane];
            }
          }
          const float w = static_cast<float>(a.coef[s] * a.inv_n);
#pragma unroll
          for (int u = 0; u < U; ++u)
            spin_term(mode[u], a.tau_hi[s], a.tau_lo[s], w, zf, inv_hbar, s0[u], s1[u], acc0[u], acc1[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int slot = slots.slot(m0 + u);
          b0[slot] = acc0[u];
          b1[slot] = acc1[u];
        }
      }
      pair_sync();
#pragma unroll
      for (int m = 0; m < V; ++m) v[m] = buf[slots.slot(m)];
    }
  }
#pragma unroll
  for (int m = 0; m < V; ++m) out[own + m * M] = v[m];
}

// The site step of the single configuration (ifrk_sites_batched: ifrk_sites_single's arithmetic,
// expression for expression) on a thread's own sites, parked in its slots of the exchange buffer:
// U sites at a time, every load of the batch before its first result.  Sites are addressed by
// 32-bit byte offsets from block-uniform bases (a member of a 4096^2 grid ends below 2^28 bytes),
// which keeps the loop's addresses out of the register file.  U = 2: four sites a batch spill at 64
// registers (a fixed step of 8 x 512^2: 307 us against 334 with four sites and half the warps, and
// 421 with four sites and 64-bit addresses).
template <int N, int V, int MODE, int TERMS, int U>
__device__ __forceinline__ void own_sites_single(float2* buf, int C, int t, int x, const IfrkColArgs& a,
                                                 const SplitConst<float>& k, long long mbase,
                                                 const float* n0, float* dn_out, float* n_out,
                                                 float2* psi_start, float2* psi_new, const float* pm,
                                                 const float* vm, float s0,
                                                 const PhiloxCellPrefix& prefix) {
  constexpr int M = RegFft<N, V>::M;
  const OwnSlots<N, V> slots(t);
  const float* nm = n0 + mbase;
#pragma unroll 1
  for (int m0 = 0; m0 < V; m0 += U) {
    unsigned o[U];
    float nv[U], acc[U], pp[U], vre[U], vim[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      o[u] = static_cast<unsigned>((t + M * (m0 + u)) * a.nx + x);
      nv[u] = at_offset(nm, 4u * o[u]);
      acc[u] = 0.f;
      if (MODE == 0) {
        pp[u] = at_offset(pm, 4u * o[u]);
        vre[u] = vim[u] = 0.f;
        if (vm) {
          if (a.potential == 2) {
            const float2 pot = at_offset(reinterpret_cast<const float2*>(vm), 8u * o[u]);
            vre[u] = pot.x;
            vim[u] = pot.y;
          } else {
            vre[u] = at_offset(vm, 4u * o[u]);
          }
        }
      }
    }
    float dv[TERMS > 0 ? TERMS : 1][U];
#pragma unroll
    for (int j = 0; j < TERMS; ++j)
#pragma unroll
      for (int u = 0; u < U; ++u)
        dv[j][u] = at_offset(static_cast<const float*>(a.dn[j]) + mbase, 4u * o[u]);
#pragma unroll
    for (int j = 0; j < TERMS; ++j)
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u] += static_cast<float>(a.coef[j]) * dv[j][u];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int slot = slots.slot(m0 + u) * C;
      float2 v = buf[slot];
      float nval = nv[u] + acc[u];
      if (MODE == 0) {
        const float rho = v.x * v.x + v.y * v.y;
        if (psi_start) at_offset(psi_start + mbase, 8u * o[u]) = v;
        const float eff = vre[u] + k.g_C * rho + k.g_R * nval;
        const float e_over = eff * k.inv_hbar;
        const float g = 0.5f * (k.R * nval - k.gamma_C) + vim[u] * k.inv_hbar;
        buf[slot] = make_float2(g * v.x + e_over * v.y, g * v.y - e_over * v.x);
        at_offset(dn_out + mbase, 4u * o[u]) = mul_rn_i(s0, pp[u]) - (k.gamma_R + k.R * rho) * nval;
      } else {
        nval = nval > 0.f ? nval : 0.f;
        at_offset(n_out + mbase, 4u * o[u]) = nval;
        if (a.noise) {
          const uint32_t cell[1] = {o[u]};
          Words4 w[1];
          philox_cells(cell, prefix, w);
          WignerDraw<float>::apply(w[0], k.noise_a + k.noise_b * nval, v.x, v.y);
          buf[slot] = v;
        }
        at_offset(psi_new + mbase, 8u * o[u]) = v;
      }
    }
  }
}

template <int N, int V, int U0, int U1>
__device__ __forceinline__ void own_sites_run(float2* buf, int C, int t, int x, const IfrkColArgs& a,
                                              const SplitConst<float>& k, long long mbase, const float* n0,
                                              float* dn_out, float* n_out, float2* psi_start,
                                              float2* psi_new, const float* pm, const float* vm, float s0,
                                              const PhiloxCellPrefix& prefix) {
  switch (a.mode * 8 + a.terms) {
#define PG_OWN(MODE, TERMS, U)                                                                          \
  case MODE * 8 + TERMS:                                                                                \
    own_sites_single<N, V, MODE, TERMS, U>(buf, C, t, x, a, k, mbase, n0, dn_out, n_out, psi_start,     \
                                           psi_new, pm, vm, s0, prefix);                                \
    break;
    PG_OWN(0, 0, U0)
    PG_OWN(0, 1, U0)
    PG_OWN(0, 2, U0)
    PG_OWN(0, 3, U0)
    PG_OWN(0, 4, U0)
    PG_OWN(0, 5, U0)
    PG_OWN(1, 1, U1)
    PG_OWN(1, 2, U1)
    PG_OWN(1, 3, U1)
    PG_OWN(1, 4, U1)
    PG_OWN(1, 5, U1)
#undef PG_OWN
    default:
      break;
  }
}

// Reservoir values of a site, n0 + sum_j coef_j dn_j on each of NQ planes, with every load issued
// before the first sum (up to TERMS + 1 loads a plane in flight).
template <int NQ>
__device__ __forceinline__ void stage_reservoirs(const IfrkColArgs& a, const float* n0,
                                                 const long long (&ridx)[4], float (&nval)[4],
                                                 float (&dsum)[4]) {
  float base[4], d[4][kIfrkMaxStages];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    base[q] = n0[ridx[q]];
#pragma unroll
    for (int j = 0; j < kIfrkMaxStages; ++j)
      d[q][j] = j < a.terms ? static_cast<const float*>(a.dn[j])[ridx[q]] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < kIfrkMaxStages; ++j)
      if (j < a.terms) acc += static_cast<float>(a.coef[j]) * d[q][j];
    dsum[q] = acc;
    nval[q] = base[q] + acc;
  }
}

// SINGLE: ifrk_sites_batched holds (kernels apart, so that neither path pays the other's registers).
template <int N, int V, int COMPS, bool SINGLE>
__global__ void __launch_bounds__(ColShape<N, V, COMPS>::MAX_THREADS,
                                  (ColShape<N, V, COMPS>::MIN_BLOCKS + COMPS - 1) / COMPS)
    ifrk_col_reg_kernel(float2* __restrict__ psi, const float* __restrict__ n0,
                        float* __restrict__ dn_out, float* __restrict__ n_out,
                        float2* __restrict__ psi_start, float2* __restrict__ psi_new,
                        const float* __restrict__ pump, const float* __restrict__ potential,
                        const float4* __restrict__ tab, const SplitConst<float>* __restrict__ consts,
                        const float* __restrict__ scales,
                        const unsigned long long* __restrict__ step_base, double* __restrict__ partials,
                        const __grid_constant__ IfrkColArgs a) {
  constexpr int M = RegFft<N, V>::M;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  const int C = a.cols, CC = C * COMPS;
  const int lcc = a.log2cols + (COMPS == 2 ? 1 : 0);
  const int c2 = threadIdx.x & (CC - 1), t = threadIdx.x >> lcc;
  const int comp = COMPS == 2 ? c2 >> a.log2cols : 0, c = c2 & (C - 1);
  const int member = blockIdx.z;
  const int nx = a.nx;
  const int x = blockIdx.x * C + c;
  float2* buf = reinterpret_cast<float2*>(smem_raw) + c2;
  const long long plane = static_cast<long long>(nx) * N;
  const long long fbase = static_cast<long long>(member) * COMPS * plane;
  float2* d = psi + fbase + comp * plane + x;
  double local = 0.0;
  float2 v[V];
#pragma unroll
  for (int m = 0; m < V; ++m) v[m] = d[static_cast<long long>(t + M * m) * nx];
  // Phase 0: the inverse transform and the site step; phase 1: the forward transform.
#pragma unroll 1
  for (int ph = 0; ph < 2; ++ph) {
    if (ph == 0 ? a.inverse : a.forward) {
      if (ph == 0) conj_all(v);
      fft_forward<N, V>(v, t, buf, CC, tab, BlockSync{});
      if (ph == 0) conj_all(v);
    }
    if (ph == 1 || a.mode == 3) continue;
    const OwnSlots<N, V> slots(t);
#pragma unroll
    for (int m = 0; m < V; ++m) buf[slots.slot(m) * CC] = v[m];
    const SplitConst<float> k = consts[member];
    const int L = a.pump_terms > 1 ? a.pump_terms : 1;
    const float* cs =
        scales ? scales + static_cast<long long>(a.scale_index * L) * a.members + member : nullptr;
    const float s0 = cs ? cs[0] : 0.f;
    const float* pm = pump + member * a.pump_stride;
    const float* vm =
        potential ? potential + member * a.pot_stride * (a.potential == 2 ? 2 : 1) : nullptr;
    const unsigned long long step = a.noise ? step_base[0] + a.step_offset : 0ull;
    const PhiloxCellPrefix prefix[2] = {
        philox_cell_prefix(static_cast<uint32_t>(step), static_cast<uint32_t>(step >> 32), 1u,
                           static_cast<uint32_t>(k.seed), static_cast<uint32_t>(k.seed >> 32)),
        philox_cell_prefix(static_cast<uint32_t>(step), static_cast<uint32_t>(step >> 32), 2u,
                           static_cast<uint32_t>(k.seed), static_cast<uint32_t>(k.seed >> 32))};
    if constexpr (SINGLE) {
      own_sites_run<N, V, 2, 2>(buf, CC, t, x, a, k, member * plane, n0, dn_out, n_out, psi_start,
                                        psi_new, pm, vm, s0, prefix[0]);
    } else {
      const IfrkGeneral<float> general{a,     k,      s0,        cs,      pm,    vm,    n0, dn_out,
                                       n_out, psi_start, psi_new, fbase, plane, prefix};
      const int Cr = a.res_comps, NQ = a.res_fields * Cr;
      const long long qstride = static_cast<long long>(Cr) * plane;
      const long long fstride = static_cast<long long>(a.members) * qstride;
      if (COMPS == 2) __syncthreads();
      float2* b0 = buf - comp * C;
      constexpr int kMine = V / COMPS;
#pragma unroll 1
      for (int h = 0; h < kMine; ++h) {
        const int m = comp * kMine + h;
        const long long o = static_cast<long long>(t + M * m) * nx + x;
        const int slot = slots.slot(m) * CC;
        float2 w[2];
        w[0] = b0[slot];
        w[1] = COMPS == 2 ? b0[slot + C] : make_float2(0.f, 0.f);
        float nval[4] = {0.f, 0.f, 0.f, 0.f}, dsum[4] = {0.f, 0.f, 0.f, 0.f};
        long long ridx[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int f = Cr == 2 ? (q >> 1) : q, cr = Cr == 2 ? (q & 1) : 0;
          ridx[q] = f * fstride + member * qstride + cr * plane + o;
        }
        const auto site = general.load(o);
        if (COMPS == 2 && NQ == 4)
          stage_reservoirs<4>(a, n0, ridx, nval, dsum);
        else if (NQ == 2)
          stage_reservoirs<2>(a, n0, ridx, nval, dsum);
        else if (NQ == 1)
          stage_reservoirs<1>(a, n0, ridx, nval, dsum);
        general.apply(w, nval, dsum, site, ridx, o, local);
        if (a.mode == 0 || (a.mode == 1 && a.noise)) {
          b0[slot] = w[0];
          if (COMPS == 2) b0[slot + C] = w[1];
        }
      }
      if (COMPS == 2) __syncthreads();
    }
    if (a.mode == 2 || (a.mode == 1 && !a.forward)) break;
#pragma unroll
    for (int m = 0; m < V; ++m) v[m] = buf[slots.slot(m) * CC];
  }
  if (a.mode == 2) {
    // Block reduction of the FP64 partial sums; one value per (member, panel).
    for (int off = 16; off > 0; off >>= 1) local += __shfl_down_sync(0xffffffffu, local, off);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = local;
    __syncthreads();
    if (warp == 0) {
      const int nw = (blockDim.x + 31) >> 5;
      double s = lane < nw ? red[lane] : 0.0;
      for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
      if (lane == 0) partials[member * gridDim.x + blockIdx.x] = s;
    }
    return;
  }
  if (a.mode == 1 && !a.forward) return;
#pragma unroll
  for (int m = 0; m < V; ++m) d[static_cast<long long>(t + M * m) * nx] = v[m];
}

template <int N, int V, int COMPS>
cudaError_t configure_row() {
  using S = RowShape<N, V, COMPS>;
  return cudaFuncSetAttribute(ifrk_row_reg_kernel<N, V, COMPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(S::MAX_THREADS / S::M * S::STRIDE * sizeof(float2)));
}
template <int N, int V, int COMPS>
cudaError_t configure_col() {
  using S = ColShape<N, V, COMPS>;
  const int smem = static_cast<int>(S::MAX_COLS * COMPS * S::SLOTS * sizeof(float2));
  const cudaError_t e = cudaFuncSetAttribute(ifrk_col_reg_kernel<N, V, COMPS, false>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess || COMPS == 2) return e;
  return cudaFuncSetAttribute(ifrk_col_reg_kernel<N, V, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              smem);
}

template <int COMPS>
cudaError_t configure(int nx, int ny) {
  auto row = [&]() -> cudaError_t {
#define PG_X(N, V) return configure_row<N, V, COMPS>()
    PG_REG_SIZES(nx, PG_X)
    return cudaErrorInvalidValue;
#undef PG_X
  };
  auto col = [&]() -> cudaError_t {
#define PG_X(N, V) return configure_col<N, V, COMPS>()
    PG_REG_SIZES(ny, PG_X)
    return cudaErrorInvalidValue;
#undef PG_X
  };
  if (reg_fft_size(nx)) {
    const cudaError_t e = row();
    if (e != cudaSuccess) return e;
  }
  return reg_fft_size(ny) ? col() : cudaSuccess;
}

template <int COMPS>
cudaError_t launch_row(const float* in, float* save, float* out, const float* tables, const float* tab,
                       IfrkRowArgs a, int sm_count, cudaStream_t stream) {
#define PG_X(N, V)                                                                                     \
  {                                                                                                    \
    using S = RowShape<N, V, COMPS>;                                                                   \
    a.rows = row_shape_rows<N, V, COMPS>(a.ny, a.members, sm_count);                                   \
    ifrk_row_reg_kernel<N, V, COMPS><<<dim3(a.ny / a.rows, 1, a.members), a.rows * S::GROUP,           \
                                       static_cast<size_t>(a.rows) * COMPS * S::STRIDE * sizeof(float2), \
                                       stream>>>(                                                      \
        reinterpret_cast<const float2*>(in), reinterpret_cast<float2*>(save),                          \
        reinterpret_cast<float2*>(out), reinterpret_cast<const float2*>(tables),                       \
        reinterpret_cast<const float4*>(tab), a);                                                      \
    return cudaGetLastError();                                                                         \
  }
  PG_REG_SIZES(a.nx, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

template <int COMPS>
cudaError_t launch_col(float* psi, const float* n0, float* dn_out, float* n_out, const float* psi_start,
                       const float* psi_new, const float* pump, const float* potential, const float* tab,
                       const SplitConst<float>* consts, const float* scales,
                       const unsigned long long* step_base, double* partials, IfrkColArgs a, int sm_count,
                       cudaStream_t stream) {
#define PG_X(N, V)                                                                                     \
  {                                                                                                    \
    a.cols = col_shape_cols<N, V, COMPS>(a.nx, a.members, sm_count);                            \
    a.log2cols = log2_of(a.cols);                                                                      \
    const dim3 grid(a.nx / a.cols, 1, a.members);                                                      \
    const int threads = a.cols * COMPS * RegFft<N, V>::M;                                              \
    const size_t smem = static_cast<size_t>(a.cols) * COMPS * RegFft<N, V>::SLOTS * sizeof(float2);    \
    auto kern = COMPS == 1 && (a.mode == 3 || ifrk_sites_batched(a)) ? ifrk_col_reg_kernel<N, V, 1, true> \
                                                                     : ifrk_col_reg_kernel<N, V, COMPS, false>; \
    kern<<<grid, threads, smem, stream>>>(                                                             \
        reinterpret_cast<float2*>(psi), n0, dn_out, n_out,                                             \
        reinterpret_cast<float2*>(const_cast<float*>(psi_start)),                                      \
        reinterpret_cast<float2*>(const_cast<float*>(psi_new)), pump, potential,                       \
        reinterpret_cast<const float4*>(tab), consts, scales, step_base, partials, a);                 \
    return cudaGetLastError();                                                                         \
  }
  PG_REG_SIZES(a.ny, PG_X)
  return cudaErrorInvalidValue;
#undef PG_X
}

}  // namespace

cudaError_t configure_ifrk_reg(int nx, int ny, int comps) {
  return comps == 2 ? configure<2>(nx, ny) : configure<1>(nx, ny);
}

int ifrk_reg_panels(int nx, int ny, int comps, int members, int sm_count) {
#define PG_X(N, V)                                                                 \
  return nx / (comps == 2 ? col_shape_cols<N, V, 2>(nx, members, sm_count)  \
                          : col_shape_cols<N, V, 1>(nx, members, sm_count))
  PG_REG_SIZES(ny, PG_X)
#undef PG_X
  return 0;
}

cudaError_t launch_ifrk_row_reg(const float* in, float* save, float* out, const float* tables,
                                const float* tab, const IfrkRowArgs& a, int sm_count,
                                cudaStream_t stream) {
  return a.comps == 2 ? launch_row<2>(in, save, out, tables, tab, a, sm_count, stream)
                      : launch_row<1>(in, save, out, tables, tab, a, sm_count, stream);
}

cudaError_t launch_ifrk_col_reg(float* psi, const float* n0, float* dn_out, float* n_out,
                                const float* psi_start, const float* psi_new, const float* pump,
                                const float* potential, const float* tab,
                                const SplitConst<float>* consts, const float* scales,
                                const unsigned long long* step_base, double* partials,
                                const IfrkColArgs& a, int sm_count, cudaStream_t stream) {
  return a.comps == 2 ? launch_col<2>(psi, n0, dn_out, n_out, psi_start, psi_new, pump, potential, tab,
                                      consts, scales, step_base, partials, a, sm_count, stream)
                      : launch_col<1>(psi, n0, dn_out, n_out, psi_start, psi_new, pump, potential, tab,
                                      consts, scales, step_base, partials, a, sm_count, stream);
}

}  // namespace pg
