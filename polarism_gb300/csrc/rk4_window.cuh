// Fused RK4 step for FP32 rows of any length: the full-width kernel's schedule (rk4_wide.cu) over a
// window of columns that need not be a power of two nor aligned for bulk copies.
//
// A block streams down a window of at most WMAX columns, two columns a thread.  A row that fits is
// one window, closed on itself; a longer row is cut into bands whose windows carry four halo
// columns on each side (the four stages each reach one column further).  Rows of psi, n_R, the
// envelope and a real potential arrive in an 8-row shared ring, three rows ahead, by cp.async of
// each thread's own two columns: 16 + 8 + 8 bytes on even row lengths, single elements on odd
// ones, so no row length is refused for its alignment.  On iteration i a thread evaluates stage
// 1 on row r-1, stage 2 on r-2, stage 3 on r-3, stage 4 and the combine on r-4; vertical
// neighbours live in registers, horizontal ones in the ring (stage 1) or one double-buffered
// exchange a row (stages 2-4).
//
// Visibility: a thread waits for its own copy of row r + 1 before it arrives at the end of the
// iteration, so stage 1, which reads its neighbours' columns of row r - 1 before it has waited for
// the previous iteration's arrivals, reads rows that landed before an earlier barrier; of row r it
// reads its own columns only.
//
// The arithmetic per site is rk4_site.cuh's, in the same order: bit for bit the streaming kernel's
// and the full-width kernel's.
#pragma once
#include <algorithm>

#include "philox.cuh"
#include "pg_internal.h"
#include "rk4_site.cuh"
#include "tma.cuh"
#include "window_internal.h"

namespace pg {
namespace {

constexpr int kWinRing = 8;  // rows resident: r-4..r plus three in flight

// Windows of at most 512 threads' worth of columns an SM (128 registers a thread).
template <int WMAX>
struct WindowShape {
  static constexpr int THREADS = WMAX / 2;
  static constexpr int BLOCKS = 512 / THREADS;  // an SM
};

// POT: 0 none, 1 real through the ring, 2 complex (or real with two lasers) from global memory.
template <int WMAX, int TERMS, int POT>
constexpr size_t window_smem() {
  return static_cast<size_t>(kWinRing) * WMAX * (12 + 4 * TERMS + (POT == 1 ? 4 : 0)) +
         static_cast<size_t>(6) * (WMAX / 2) * 16 + sizeof(uint64_t);
}

template <int WMAX, bool NOISE, bool GENERAL, int POT, int TERMS>
__global__ void __launch_bounds__(WindowShape<WMAX>::THREADS, WindowShape<WMAX>::BLOCKS)
    rk4_window_kernel(const float2* __restrict__ psi_in, const float* __restrict__ n_in,
                      const float* __restrict__ pump, float2* __restrict__ psi_out,
                      float* __restrict__ n_out, const RhsConst<float>* __restrict__ consts,
                      const float* __restrict__ scales,
                      const unsigned long long* __restrict__ step_base, const int step_offset,
                      const float dt, const WindowGeom g, int* __restrict__ err_flag) {
  constexpr int HALF = WMAX / 2;  // exchange-buffer stride
  // Rows meet at a block-wide barrier, but for one block an SM with a complex potential: its loads from
  // global memory stall the warps unevenly, and a split arrive/wait barrier lets them drift apart by up to
  // a row (8 x 1020^2 125 us a step against 138; without a potential 63 against 59).  Each warp arrives once: an
  // arrival of all its lanes counts as 32 at once, and where a wait had given up, more arrivals than a phase
  // still expects, which is an error of the barrier; one at a time they only move on to the next phase.
  constexpr bool kSplit = WindowShape<WMAX>::BLOCKS == 1 && POT == 2 && TERMS == 1;
  if (g.halt != nullptr && __ldcg(g.halt) != 0) return;  // steady-state monitor halted the run
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2* ring_psi = reinterpret_cast<float2*>(smem_raw);                 // [kWinRing][WMAX]
  float* ring_n = reinterpret_cast<float*>(ring_psi + kWinRing * WMAX);   // [kWinRing][WMAX]
  float* ring_p = ring_n + kWinRing * WMAX;                               // [kWinRing][TERMS][WMAX]
  float* ring_v = ring_p + kWinRing * TERMS * WMAX;                       // [kWinRing][WMAX] (POT 1)
  float2* xa = reinterpret_cast<float2*>(ring_v + (POT == 1 ? kWinRing * WMAX : 0));  // [2][3][HALF]
  float2* xb = xa + 6 * HALF;                                             // [2][3][HALF]
  const uint32_t xbar = smem_u32(xb + 6 * HALF);

  const int nx = g.nx, ny = g.ny;
  const int t = threadIdx.x;
  const bool closed = g.bands == 1;
  const bool odd = (nx & 1) != 0;
  const int w = closed ? nx : g.band_w + 8;       // window columns
  const int active = (w + 1) >> 1;                // threads that own columns
  const bool owner = t < active;                  // the others copy, publish and write nothing
  const int tc = min(t, active - 1);
  const int col0 = 2 * tc;
  // Ring columns left of the thread's first and right of its second column.  A closed window of odd
  // length gives its last thread a second column that repeats column 0.
  const bool first = tc == 0, last = tc == active - 1;
  const int lcol = first ? (closed ? nx - 1 : 0) : col0 - 1;
  const int rcol = last ? (closed ? (odd ? 1 : 0) : w - 1) : col0 + 2;
  const float2* lsrc = first ? (closed ? (odd ? xa : xb) + active - 1 : xb) : xb + tc - 1;
  const float2* rsrc = last ? (closed ? (odd ? xb : xa) : xa + tc) : xa + tc + 1;
  const long long plane = static_cast<long long>(nx) * ny;

  if (kSplit && t == 0) {
    mbar_init(xbar, blockDim.x / 32);
    fence_mbar_init();
  }

  const long long total_rows = static_cast<long long>(g.members) * g.bands * ny;
  const long long r_begin = total_rows * blockIdx.x / gridDim.x;
  const long long r_end = total_rows * (blockIdx.x + 1) / gridDim.x;
  const float hh = 0.5f * dt, h6 = dt / 6.0f, h3 = dt / 3.0f;
  unsigned it = 0;  // iterations so far
  bool timed_out = false;

  long long gr = r_begin;
  while (gr < r_end) {
    // Row space [member][band][row]; a segment stays within one (member, band).
    const long long unit = gr / ny;
    const int member = static_cast<int>(unit / g.bands);
    const int band = static_cast<int>(unit % g.bands);
    const int ya = static_cast<int>(gr - unit * ny);
    const int yb = static_cast<int>(min(static_cast<long long>(ny), ya + (r_end - gr)));
    gr += yb - ya;
    const int h_rows = yb - ya;
    const int n_iter = h_rows + 8;

    const RhsConst<float> kk = consts[member];
    const WideConst k = wide_const(kk);
    float cs[3][TERMS];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int l = 0; l < TERMS; ++l)
        cs[q][l] = scales[(static_cast<long long>(step_offset * 3 + q) * TERMS + l) * g.members + member];
    // With one laser a stage multiplies s_q by the envelope; with several, pump_pair forms
    // sum_l c_ql E_l and the stage's factor is 1 (a multiply by 1 rounds nothing).
    const float s0 = TERMS == 1 ? cs[0][0] : 1.f;
    const float s1 = TERMS == 1 ? cs[1][0] : 1.f;
    const float s2 = TERMS == 1 ? cs[2][0] : 1.f;
    const unsigned long long noise_step = NOISE ? step_base[0] + step_offset : 0ull;
    const PhiloxCellPrefix prefix =
        philox_cell_prefix(static_cast<uint32_t>(noise_step), static_cast<uint32_t>(noise_step >> 32),
                           1u, static_cast<uint32_t>(kk.seed), static_cast<uint32_t>(kk.seed >> 32));
    // Grid columns of the thread's two window columns.
    const int x0 = band * g.band_w;
    int ga = (closed ? 0 : x0 - 4) + col0;
    ga = ga < 0 ? ga + nx : (ga >= nx ? ga - nx : ga);
    const int gb = ga + 1 == nx ? 0 : ga + 1;
    const int bw = min(g.band_w, nx - x0);  // columns this band writes
    const bool wa = owner && (closed || (col0 >= 4 && col0 < 4 + bw));
    const bool wb = owner && (closed ? col0 + 1 < nx : (col0 + 1 >= 4 && col0 + 1 < 4 + bw));
    const float2* psi_m = psi_in + member * plane;
    const float* n_m = n_in + member * plane;
    const float* p_m = pump + member * g.pump_stride;
    const float* pot_m =
        POT != 0 && g.pot != nullptr ? g.pot + member * g.pot_stride * (g.pot_kind == 2 ? 2 : 1) : nullptr;
    auto pot_at = [&](int row, int slot, float2& va, float2& vb) {
      va = vb = make_float2(0.f, 0.f);
      if (POT == 1) {
        const float2 v = *reinterpret_cast<const float2*>(ring_v + slot * WMAX + col0);
        va.x = v.x;
        vb.x = v.y;
      } else if (POT == 2 && pot_m != nullptr) {
        const long long oa = static_cast<long long>(row) * nx + ga, ob = static_cast<long long>(row) * nx + gb;
        if (g.pot_kind == 2) {
          va = *reinterpret_cast<const float2*>(pot_m + 2 * oa);
          vb = *reinterpret_cast<const float2*>(pot_m + 2 * ob);
        } else {
          va.x = pot_m[oa];
          vb.x = pot_m[ob];
        }
      }
    };
    auto rhs2 = [&](float2 ca, float2 cb, float2 L, float2 R, float2 upa, float2 upb, float2 dna,
                    float2 dnb, float2 n2, float s, float2 P, float2 va, float2 vb, float2& da,
                    float2& db) -> float2 {
      if (GENERAL) {
        const bool rl = g.relax != 0;
        const float x = site_rhs_general(ca, L, cb, upa, dna, n2.x, __fmul_rn(s, P.x), k, va.x, va.y, rl, da);
        const float y = site_rhs_general(cb, ca, R, upb, dnb, n2.y, __fmul_rn(s, P.y), k, vb.x, vb.y, rl, db);
        return make_float2(x, y);
      }
      return pair_rhs(ca, cb, L, R, upa, upb, dna, dnb, n2, __fmul2_rn(make_float2(s, s), P), k, da, db);
    };
    auto pump_pair = [&](int slot, int q) -> float2 {
      const float* base = ring_p + slot * TERMS * WMAX + col0;
      const float2 e0 = *reinterpret_cast<const float2*>(base);
      if (TERMS == 1) return e0;
      float2 v = make_float2(__fmul_rn(cs[q][0], e0.x), __fmul_rn(cs[q][0], e0.y));
#pragma unroll
      for (int l = 1; l < TERMS; ++l) {
        const float2 e = *reinterpret_cast<const float2*>(base + l * WMAX);
        v = make_float2(__fadd_rn(v.x, __fmul_rn(cs[q][l], e.x)), __fadd_rn(v.y, __fmul_rn(cs[q][l], e.y)));
      }
      return v;
    };
    int row_load = ya - 4;  // row of the next copy
    while (row_load < 0) row_load += ny;
    // Copies of the thread's columns of the next row into ring slot `slot`.
    auto issue = [&](int slot) {
      const int o = row_load * nx;
      row_load = row_load + 1 == ny ? 0 : row_load + 1;
      if (!owner) return;
      float2* dpsi = ring_psi + slot * WMAX + col0;
      float* dn = ring_n + slot * WMAX + col0;
      float* dp = ring_p + slot * TERMS * WMAX + col0;
      float* dv = ring_v + slot * WMAX + col0;
      if (!odd) {
        cp_async16(dpsi, psi_m + o + ga);
        cp_async8(dn, n_m + o + ga);
#pragma unroll
        for (int l = 0; l < TERMS; ++l) cp_async8(dp + l * WMAX, p_m + l * g.pump_term_stride + o + ga);
        if (POT == 1) cp_async8(dv, pot_m + o + ga);
      } else {
        cp_async8(dpsi, psi_m + o + ga);
        cp_async8(dpsi + 1, psi_m + o + gb);
        cp_async4(dn, n_m + o + ga);
        cp_async4(dn + 1, n_m + o + gb);
#pragma unroll
        for (int l = 0; l < TERMS; ++l) {
          cp_async4(dp + l * WMAX, p_m + l * g.pump_term_stride + o + ga);
          cp_async4(dp + l * WMAX + 1, p_m + l * g.pump_term_stride + o + gb);
        }
        if (POT == 1) {
          cp_async4(dv, pot_m + o + ga);
          cp_async4(dv + 1, pot_m + o + gb);
        }
      }
    };
    // Every read of the previous segment's ring and exchange is done before the first copy.
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      issue(i);
      cp_async_commit();
    }

    Pair q1[4], q2[4], q3[4], acc[4];
    float2 m1[4], m2[4], m3[4], accn[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      q1[s] = q2[s] = q3[s] = acc[s] = Pair{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      m1[s] = m2[s] = m3[s] = accn[s] = make_float2(0.f, 0.f);
    }
    int row_out = ya - 8;
    while (row_out < 0) row_out += ny;
    cp_async_wait<2>();

#pragma unroll 1
    for (int i0 = 0; i0 < n_iter; i0 += kWinRing) {
#pragma unroll
      for (int j = 0; j < kWinRing; ++j) {
        const int i = i0 + j;
        if (i >= n_iter) break;
        const int ja = (j + 3) & 3, jb = (j + 2) & 3, jc = (j + 1) & 3, jd = j & 3;
        const int slot0 = j, slot1 = (j + 7) % 8, slot2 = (j + 6) % 8, slot3 = (j + 5) % 8, slot4 = (j + 4) % 8;
        // Stage 1 at row r-1 from the ring: k1 = f(psi0).
        const float2* R1 = ring_psi + slot1 * WMAX;
        const float4 c4 = *reinterpret_cast<const float4*>(R1 + col0);
        const float4 u4 = *reinterpret_cast<const float4*>(ring_psi + slot2 * WMAX + col0);
        const float4 d4 = *reinterpret_cast<const float4*>(ring_psi + slot0 * WMAX + col0);
        const float2 lt = R1[lcol], rt = R1[rcol];
        const float2 c0 = make_float2(c4.x, c4.y), c1 = make_float2(c4.z, c4.w);
        const float2 up0 = make_float2(u4.x, u4.y), up1 = make_float2(u4.z, u4.w);
        const float2 dn0 = make_float2(d4.x, d4.y), dn1 = make_float2(d4.z, d4.w);
        const float2 n1v = *reinterpret_cast<const float2*>(ring_n + slot1 * WMAX + col0);
        const float2 P1 = pump_pair(slot1, 0);
        int srow[4] = {0, 0, 0, 0};  // rows of the four stages (potential in global memory)
        if (POT == 2) {
          srow[3] = row_out;
#pragma unroll
          for (int q = 2; q >= 0; --q) srow[q] = srow[q + 1] + 1 == ny ? 0 : srow[q + 1] + 1;
        }
        {
          float2 da, db, va, vb;
          pot_at(srow[0], slot1, va, vb);
          const float2 dn2 = rhs2(c0, c1, lt, rt, up0, up1, dn0, dn1, n1v, s0, P1, va, vb, da, db);
          q1[ja] = Pair{axpy2(hh, da, c0), axpy2(hh, db, c1)};
          acc[ja] = Pair{axpy2(h6, da, c0), axpy2(h6, db, c1)};
          m1[ja] = axpy2(hh, dn2, n1v);
          accn[ja] = axpy2(h6, dn2, n1v);
        }
        if (kSplit) {
          // Every thread has arrived at the end of iteration i-1: published its stage values there
          // and finished every read of iteration i-1.
          const unsigned gi = it + i;
          if (gi > 0 && !mbar_wait_bounded(xbar, (gi - 1) & 1u, g.wait_limit)) timed_out = true;
        }
        // Row r+3 into the slot of row r-5, whose last reader was this thread's stage 4.
        if (i + 3 < n_iter) issue((j + 3) % 8);
        cp_async_commit();
        // The draw for this iteration's output row, in the straight-line code of stages 2-4 so that
        // the integer and SFU work fills their issue gaps.
        float r2a = 0.f, sna = 0.f, csa = 0.f, r2b = 0.f, snb = 0.f, csb = 0.f;
        if (NOISE) {
          const uint32_t cells[2] = {static_cast<uint32_t>(row_out * nx + ga),
                                     static_cast<uint32_t>(row_out * nx + gb)};
          Words4 wd[2];
          philox_cells(cells, prefix, wd);
          WignerDraw<float>::prepare(wd[0], r2a, sna, csa);
          WignerDraw<float>::prepare(wd[1], r2b, snb, csb);
        }
        const int xo = ((j + 1) & 1) * 3 * HALF;
        // Stage 2 at row r-2: k2 = f(psi1).
        {
          const float2 lt2 = lsrc[xo], rt2 = rsrc[xo];
          const float2 P2 = pump_pair(slot2, 1);
          const float2 n0 = *reinterpret_cast<const float2*>(ring_n + slot2 * WMAX + col0);
          const Pair c = q1[jb];
          float2 da, db, va, vb;
          pot_at(srow[1], slot2, va, vb);
          const float2 dn2 = rhs2(c.a, c.b, lt2, rt2, q1[jc].a, q1[jc].b, q1[ja].a, q1[ja].b, m1[jb], s1, P2,
                                  va, vb, da, db);
          q2[jb] = Pair{axpy2(hh, da, up0), axpy2(hh, db, up1)};  // psi0 at row r-2
          m2[jb] = axpy2(hh, dn2, n0);
          acc[jb] = Pair{axpy2(h3, da, acc[jb].a), axpy2(h3, db, acc[jb].b)};
          accn[jb] = axpy2(h3, dn2, accn[jb]);
        }
        // Stage 3 at row r-3: k3 = f(psi2).
        {
          const float2 lt3 = lsrc[xo + HALF], rt3 = rsrc[xo + HALF];
          const float2 P3 = pump_pair(slot3, 1);
          const float2 n0 = *reinterpret_cast<const float2*>(ring_n + slot3 * WMAX + col0);
          const float4 p4 = *reinterpret_cast<const float4*>(ring_psi + slot3 * WMAX + col0);
          const Pair c = q2[jc];
          float2 da, db, va, vb;
          pot_at(srow[2], slot3, va, vb);
          const float2 dn2 = rhs2(c.a, c.b, lt3, rt3, q2[jd].a, q2[jd].b, q2[jb].a, q2[jb].b, m2[jc], s1, P3,
                                  va, vb, da, db);
          q3[jc] = Pair{axpy2(dt, da, make_float2(p4.x, p4.y)), axpy2(dt, db, make_float2(p4.z, p4.w))};
          m3[jc] = axpy2(dt, dn2, n0);
          acc[jc] = Pair{axpy2(h3, da, acc[jc].a), axpy2(h3, db, acc[jc].b)};
          accn[jc] = axpy2(h3, dn2, accn[jc]);
        }
        // Stage 4 at row r-4: k4 = f(psi3), final combine, clamp, Wigner increment.
        {
          const float2 lt4 = lsrc[xo + 2 * HALF], rt4 = rsrc[xo + 2 * HALF];
          const float2 P4 = pump_pair(slot4, 2);
          const Pair c = q3[jd];
          float2 da, db, va, vb;
          pot_at(srow[3], slot4, va, vb);
          const float2 dn2 = rhs2(c.a, c.b, lt4, rt4, q3[ja].a, q3[ja].b, q3[jc].a, q3[jc].b, m3[jd], s2, P4,
                                  va, vb, da, db);
          float2 oa = axpy2(h6, da, acc[jd].a);
          float2 ob = axpy2(h6, db, acc[jd].b);
          const float2 nab = axpy2(h6, dn2, accn[jd]);
          float na = nab.x, nb = nab.y;
          na = na < 0.f ? 0.f : na;
          nb = nb < 0.f ? 0.f : nb;
          if (wa && i >= 8) {
            const long long o = member * plane + row_out * nx + ga;
            if (NOISE) {
              WignerDraw<float>::add(fmaf(k.noise_b, na, k.noise_a), r2a, sna, csa, oa.x, oa.y);
              WignerDraw<float>::add(fmaf(k.noise_b, nb, k.noise_a), r2b, snb, csb, ob.x, ob.y);
            }
            if (!odd) {
              *reinterpret_cast<float4*>(psi_out + o) = make_float4(oa.x, oa.y, ob.x, ob.y);
              *reinterpret_cast<float2*>(n_out + o) = make_float2(na, nb);
            } else {
              psi_out[o] = oa;
              n_out[o] = na;
              if (wb) {
                psi_out[o + 1] = ob;
                n_out[o + 1] = nb;
              }
            }
          }
        }
        // Publish stage inputs for the horizontal neighbours.
        if (owner) {
          const int o = (j & 1) * 3 * HALF + tc;
          xa[o] = q1[ja].a;
          xb[o] = q1[ja].b;
          xa[o + HALF] = q2[jb].a;
          xb[o + HALF] = q2[jb].b;
          xa[o + 2 * HALF] = q3[jc].a;
          xb[o + 2 * HALF] = q3[jc].b;
        }
        row_out = row_out + 1 == ny ? 0 : row_out + 1;
        cp_async_wait<2>();  // row r + 1 has landed
        if (kSplit) {
          __syncwarp();
          if ((t & 31) == 0) mbar_arrive(xbar);
        } else {
          __syncthreads();
        }
      }
    }
    it += n_iter;
    cp_async_wait<0>();
  }
  if (timed_out) atomicOr(err_flag, 1);
}

}  // namespace
}  // namespace pg

namespace pg {
namespace {

template <int WMAX, bool NOISE, bool GENERAL, int POT, int TERMS>
cudaError_t launch_window_variant(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                                  float* n_out, const RhsConst<float>* consts, const float* scales,
                                  const unsigned long long* step_base, int step_offset, float dt,
                                  const WindowGeom& g, int* err_flag, cudaStream_t stream) {
  constexpr size_t smem = window_smem<WMAX, TERMS, POT>();
  auto kern = rk4_window_kernel<WMAX, NOISE, GENERAL, POT, TERMS>;
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  const int w = g.bands == 1 ? g.nx : g.band_w + 8;
  const int threads = ((w + 1) / 2 + 31) / 32 * 32;
  if (w + (w & 1) > WMAX || threads > WindowShape<WMAX>::THREADS) return cudaErrorInvalidConfiguration;
  kern<<<g.blocks, threads, smem, stream>>>(reinterpret_cast<const float2*>(psi_in), n_in, pump,
                                            reinterpret_cast<float2*>(psi_out), n_out, consts, scales,
                                            step_base, step_offset, dt, g, err_flag);
  return cudaGetLastError();
}

}  // namespace

template <int WMAX>
cudaError_t launch_window_t(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                            float* n_out, const RhsConst<float>* consts, const float* scales,
                            const unsigned long long* step_base, int step_offset, float dt, bool noise,
                            const WindowGeom& g, int* err_flag, cudaStream_t stream) {
#define PG_WIN(G, P, L)                                                                            \
  (noise ? launch_window_variant<WMAX, true, G, P, L>(psi_in, n_in, pump, psi_out, n_out, consts,  \
                                                      scales, step_base, step_offset, dt, g,       \
                                                      err_flag, stream)                            \
         : launch_window_variant<WMAX, false, G, P, L>(psi_in, n_in, pump, psi_out, n_out, consts, \
                                                       scales, step_base, step_offset, dt, g,      \
                                                       err_flag, stream))
  if (g.pump_terms == 2) return PG_WIN(true, 2, 2);
  if (g.pump_terms != 1) return cudaErrorInvalidValue;
  if (g.pot_kind == 2) return PG_WIN(true, 2, 1);
  if (g.pot_kind == 1) return PG_WIN(true, 1, 1);
  return g.relax ? PG_WIN(true, 0, 1) : PG_WIN(false, 0, 1);
#undef PG_WIN
}

}  // namespace pg
