// Whole-step RK4 on two-dimensional tiles (any grid size, both precisions, every option of the
// streaming kernel of rk4.cu, the same bits per site).
//
// A block advances one TW x TH tile of one member through the four stages in shared memory.
// Stage s = 1..4 is needed on the tile grown by 4 - s sites on each side, so a tile costs
// sum_s (TW + 2 (4 - s)) (TH + 2 (4 - s)) site-stages for 4 TW TH useful ones, whatever the grid:
// 1.75 times the useful work at 16 x 8 counted in whole warps, 1.34 at 32 x 16, 1.22 at 32 x 32.
// The streaming kernel runs all four stages on every row of its 8-row fill instead.
//
// Work is dealt in units of 32 sites.  The tile's own sites are fixed to threads (their RK4
// accumulators stay in registers); the ring of each stage is enumerated compactly over the
// block's warps, so no warp runs half empty along the ring's edges.  Ring sites need no
// accumulator.  One barrier a stage.
#pragma once
#include "philox.cuh"
#include "pg_internal.h"
#include "rk4_general.cuh"

namespace pg {
namespace {

template <int TW, int TH>
struct TileShape {
  static_assert(TW * TH % 32 == 0, "the tile's own sites fill whole warps");
  static constexpr int OUT = TW * TH;
  static constexpr int OUT_UNITS = OUT / 32;
  static constexpr int W0 = TW + 8, H0 = TH + 8;  // psi0
  static constexpr int W1 = TW + 6, H1 = TH + 6;  // stage 1 and the scalars
  static constexpr int ring(int r) { return (TW + 2 * r) * (TH + 2 * r) - OUT; }
  static constexpr int ring_units(int r) { return (ring(r) + 31) / 32; }
  static constexpr int units() {
    return 4 * OUT_UNITS + ring_units(3) + ring_units(2) + ring_units(1);
  }
};

// Site e of the ring of width r around the tile: the r rows above, the r rows below, then the
// r columns on either side.
template <int TW, int TH, int R>
__device__ __forceinline__ void ring_site(int e, int& x, int& y) {
  constexpr int kWide = TW + 2 * R;
  if (e < 2 * R * kWide) {
    const int row = e / kWide;
    x = e % kWide - R;
    y = row < R ? row - R : TH + row - R;
  } else {
    const int q = e - 2 * R * kWide;
    const int c = q % (2 * R);
    y = q / (2 * R);
    x = c < R ? c - R : TW + c - R;
  }
}

template <int S>
struct StageTag {
  static constexpr int value = S;
};

__device__ __forceinline__ int wrap_index(int i, int n) {
  while (i < 0) i += n;
  while (i >= n) i -= n;
  return i;
}

template <typename T, bool TWO, int TW, int TH>
constexpr size_t tile_smem() {
  using S = TileShape<TW, TH>;
  return (static_cast<size_t>(S::W0) * S::H0 + 2 * static_cast<size_t>(S::W1) * S::H1) * 2 * sizeof(T) +
         static_cast<size_t>(S::W1) * S::H1 * (TWO ? 5 : 3) * sizeof(T);
}

template <typename T, bool NOISE, bool GENERAL, bool TWO, int TW, int TH, int WARPS, int MIN_BLOCKS>
__global__ void __launch_bounds__(WARPS * 32, MIN_BLOCKS)
    rk4_tile_kernel(const typename Cplx<T>::type* __restrict__ psi_in, const T* __restrict__ n_in,
                    const T* __restrict__ pump, const T* __restrict__ potential,
                    typename Cplx<T>::type* __restrict__ psi_out, T* __restrict__ n_out,
                    const RhsConst<T>* __restrict__ consts, const T* __restrict__ scales,
                    const unsigned long long* __restrict__ step_base, const int step_offset,
                    const T dt, const RK4Geom g, const RK4Features f) {
  using C2 = typename Cplx<T>::type;
  using S = TileShape<TW, TH>;
  constexpr int kOwn = (S::OUT_UNITS + WARPS - 1) / WARPS;  // own units of a warp
  constexpr bool two = GENERAL && TWO;
  if (g.halt != nullptr && __ldcg(g.halt) != 0) return;  // steady-state monitor halted the run
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2* p0 = reinterpret_cast<C2*>(smem_raw);  // [H0][W0], origin (-4, -4)
  C2* qa = p0 + S::W0 * S::H0;               // [H1][W1], origin (-3, -3), as everything below
  C2* qb = qa + S::W1 * S::H1;
  T* n0 = reinterpret_cast<T*>(qb + S::W1 * S::H1);
  T* env = n0 + S::W1 * S::H1;
  T* m = env + S::W1 * S::H1;   // the stage's reservoir
  T* u0 = m + S::W1 * S::H1;    // the inactive field and its stage value (two-field reservoirs)
  T* v = u0 + S::W1 * S::H1;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int member = blockIdx.z;
  const int nx = g.nx, ny = g.ny;
  const long long plane = static_cast<long long>(nx) * ny;
  const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
  const RhsConst<T> k = consts[member];
  const int L = GENERAL ? f.pump_terms : 1;
  const T* coef = scales + static_cast<long long>(step_offset * 3 * L) * g.members + member;
  const long long cstep = static_cast<long long>(L) * g.members;  // to the next stage sample
  const T sc[3] = {coef[0], coef[cstep], coef[2 * cstep]};
  const bool multi = GENERAL && L > 1;
  const T hh = dt * T(0.5), h6 = dt / T(6), h3 = dt / T(3);
  const C2* psi_m = psi_in + member * plane;
  const T* n_m = n_in + member * plane;
  const long long field2 = static_cast<long long>(g.members) * plane;
  const T* pump_m = pump + member * g.pump_stride;
  const T* pot_m = potential ? potential + member * g.pot_stride * (f.potential == 2 ? 2 : 1) : nullptr;

  for (int e = tid; e < S::W0 * S::H0; e += WARPS * 32) {
    const int y = e / S::W0, x = e % S::W0;
    const long long o = static_cast<long long>(wrap_index(y0 - 4 + y, ny)) * nx + wrap_index(x0 - 4 + x, nx);
    p0[e] = psi_m[o];
    if (y >= 1 && y < S::H0 - 1 && x >= 1 && x < S::W0 - 1) {
      const int s = (y - 1) * S::W1 + x - 1;
      n0[s] = f.reservoir ? n_m[o] : T(0);
      env[s] = pump_m[o];
      if (two) u0[s] = n_m[field2 + o];
    }
  }
  __syncthreads();

  C2 acc[kOwn];
  T accn[kOwn], accu[kOwn];

  // Stage STAGE at tile site (x, y): the right-hand side there, into d, dnr and du.
  auto rhs_at = [&](auto stage, int x, int y, C2& d, T& dnr, T& du) {
    constexpr int ST = decltype(stage)::value;
    const int s = (y + 3) * S::W1 + x + 3;
    const C2* q = ST == 1 ? p0 : (ST == 3 ? qb : qa);
    const int w = ST == 1 ? S::W0 : S::W1;
    const int at = ST == 1 ? (y + 4) * S::W0 + x + 4 : s;
    T vre = T(0), vim = T(0);
    T sP;
    if (GENERAL && (f.potential || multi)) {
      const long long o = static_cast<long long>(wrap_index(y0 + y, ny)) * nx + wrap_index(x0 + x, nx);
      if (f.potential) {
        vre = f.potential == 2 ? pot_m[2 * o] : pot_m[o];
        vim = f.potential == 2 ? pot_m[2 * o + 1] : T(0);
      }
      if (multi)
        sP = pump_terms_value(pump_m, g.pump_term_stride, coef + (ST / 2) * cstep, g.members, L, o);
    }
    if (!multi) sP = pump_mul_rn(sc[ST / 2], env[s]);
    const T n = ST == 1 ? n0[s] : m[s];
    const T n2 = two ? (ST == 1 ? u0[s] : v[s]) : T(0);
    general_rhs<T, GENERAL, TWO>(q[at], q[at - 1], q[at + 1], q[at - w], q[at + w], n, sP, k, vre, vim,
                                 f, d, dnr, n2, du);
  };
  // Stages 1-3: the next stage's values at (x, y).
  auto advance_site = [&](auto stage, int x, int y, const C2& d, T dnr, T du) {
    constexpr int ST = decltype(stage)::value;
    const int s = (y + 3) * S::W1 + x + 3;
    const T h = ST == 3 ? dt : hh;
    C2* q = ST == 2 ? qb : qa;
    q[s] = axpy_t<T>(h, d, p0[(y + 4) * S::W0 + x + 4]);
    m[s] = fma_t(h, dnr, n0[s]);
    if (two) v[s] = fma_t(h, du, u0[s]);
  };
  auto run_stage = [&](auto stage) {
    constexpr int ST = decltype(stage)::value;
    constexpr int R = 4 - ST;
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
      const int unit = warp + q * WARPS;
      if (S::OUT_UNITS % WARPS != 0 && unit >= S::OUT_UNITS) break;
      const int e = unit * 32 + lane;
      const int x = e % TW, y = e / TW;
      C2 d;
      T dnr, du;
      rhs_at(stage, x, y, d, dnr, du);
      const T ha = ST == 1 ? h6 : h3;
      if (ST == 1) {
        const int s = (y + 3) * S::W1 + x + 3;
        acc[q] = axpy_t<T>(ha, d, p0[(y + 4) * S::W0 + x + 4]);
        accn[q] = fma_t(ha, dnr, n0[s]);
        if (two) accu[q] = fma_t(ha, du, u0[s]);
      } else {
        acc[q] = axpy_t<T>(ha, d, acc[q]);
        accn[q] = fma_t(ha, dnr, accn[q]);
        if (two) accu[q] = fma_t(ha, du, accu[q]);
      }
      advance_site(stage, x, y, d, dnr, du);
    }
    // The ring's units go to the warps after those that hold the last own units.
    constexpr int kFirst = S::OUT_UNITS % WARPS;
    for (int u = warp >= kFirst ? warp - kFirst : warp + WARPS - kFirst; u < S::ring_units(R); u += WARPS) {
      const int e = u * 32 + lane;
      if (e < S::ring(R)) {
        int x, y;
        ring_site<TW, TH, R>(e, x, y);
        C2 d;
        T dnr, du;
        rhs_at(stage, x, y, d, dnr, du);
        advance_site(stage, x, y, d, dnr, du);
      }
    }
    __syncthreads();
  };
  run_stage(StageTag<1>{});
  run_stage(StageTag<2>{});
  run_stage(StageTag<3>{});

  // Stage 4, final combine, clamp, Wigner increment.
  const unsigned long long noise_step = NOISE ? step_base[0] + step_offset : 0ull;
  const PhiloxCellPrefix prefix =
      philox_cell_prefix(static_cast<uint32_t>(noise_step), static_cast<uint32_t>(noise_step >> 32),
                         1u, static_cast<uint32_t>(k.seed), static_cast<uint32_t>(k.seed >> 32));
#pragma unroll
  for (int q = 0; q < kOwn; ++q) {
    const int unit = warp + q * WARPS;
    if (S::OUT_UNITS % WARPS != 0 && unit >= S::OUT_UNITS) break;
    const int e = unit * 32 + lane;
    const int x = e % TW, y = e / TW;
    C2 d;
    T dnr, du;
    rhs_at(StageTag<4>{}, x, y, d, dnr, du);
    C2 out = axpy_t<T>(h6, d, acc[q]);
    T on = fma_t(h6, dnr, accn[q]);
    on = on < T(0) ? T(0) : on;
    if (x0 + x >= nx || y0 + y >= ny) continue;
    const long long o = static_cast<long long>(y0 + y) * nx + x0 + x;
    if (NOISE) {
      const uint32_t cell[1] = {static_cast<uint32_t>(o)};
      Words4 w[1];
      philox_cells(cell, prefix, w);
      WignerDraw<T>::apply(w[0], fma_t(k.noise_b, on, k.noise_a), out.x, out.y);
    }
    psi_out[member * plane + o] = out;
    if (!GENERAL || f.reservoir) n_out[member * plane + o] = on;
    if (two) {
      T ou = fma_t(h6, du, accu[q]);
      ou = ou < T(0) ? T(0) : ou;
      n_out[field2 + member * plane + o] = ou;
    }
  }
}

template <typename T, bool NOISE, bool GENERAL, bool TWO, int TW, int TH, int WARPS, int MIN_BLOCKS>
cudaError_t launch_tile_variant(const T* psi_in, const T* n_in, const T* pump, const T* potential,
                                T* psi_out, T* n_out, const RhsConst<T>* consts, const T* scales,
                                const unsigned long long* step_base, int step_offset, T dt,
                                const RK4Geom& g, const RK4Features& f, cudaStream_t stream) {
  using C2 = typename Cplx<T>::type;
  constexpr size_t smem = tile_smem<T, TWO, TW, TH>();
  auto kern = rk4_tile_kernel<T, NOISE, GENERAL, TWO, TW, TH, WARPS, MIN_BLOCKS>;
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((g.nx + TW - 1) / TW, (g.ny + TH - 1) / TH, g.members);
  kern<<<grid, WARPS * 32, smem, stream>>>(reinterpret_cast<const C2*>(psi_in), n_in, pump, potential,
                                           reinterpret_cast<C2*>(psi_out), n_out, consts, scales,
                                           step_base, step_offset, dt, g, f);
  return cudaGetLastError();
}

// The tile of `shape` (index into the precision's list) for the launch's features.
template <typename T, int TW, int TH, int WARPS, int MIN_BLOCKS>
cudaError_t launch_tile_shape(const T* psi_in, const T* n_in, const T* pump, const T* potential,
                              T* psi_out, T* n_out, const RhsConst<T>* consts, const T* scales,
                              const unsigned long long* step_base, int step_offset, T dt, bool noise,
                              const RK4Geom& g, const RK4Features& f, cudaStream_t stream) {
  const bool general = f.potential != 0 || f.relax != 0 || f.reservoir != 1 || f.pump_terms > 1;
  const bool two = f.reservoir >= 2;
#define PG_TILE_VARIANT(N, G, W)                                                                 \
  launch_tile_variant<T, N, G, W, TW, TH, WARPS, MIN_BLOCKS>(psi_in, n_in, pump, potential,      \
                                                             psi_out, n_out, consts, scales,     \
                                                             step_base, step_offset, dt, g, f, stream)
  if (noise) {
    if (two) return PG_TILE_VARIANT(true, true, true);
    return general ? PG_TILE_VARIANT(true, true, false) : PG_TILE_VARIANT(true, false, false);
  }
  if (two) return PG_TILE_VARIANT(false, true, true);
  return general ? PG_TILE_VARIANT(false, true, false) : PG_TILE_VARIANT(false, false, false);
#undef PG_TILE_VARIANT
}

}  // namespace
}  // namespace pg
