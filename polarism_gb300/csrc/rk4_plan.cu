// Which kernel steps a grid when the caller leaves the choice.  FP64: the tile kernel (rk4_tile_f64.cu;
// measured without / with Wigner noise, us a step, streaming kernel -> tile kernel: 92.6 -> 11.4 /
// 141 -> 14.7 at 128^2, 179 -> 24.4 / 269 -> 35.9 at 256^2, 208 -> 78 / 314 -> 123 at 512^2,
// 310 -> 268 / 495 -> 426 at 1024^2), where its launch fits.  FP32: the tile kernel (rk4_tile.cuh),
// the window kernel (rk4_window.cuh), the full-width kernel (rk4_wide.cu) or the streaming kernel
// (rk4.cu).  All give the same bits, so the choice is the smallest modelled time.
//
// The models (us a step, fitted to measurements with Wigner noise; without it every kernel takes
// about 0.7 of them) and what they were fitted on:
//   tile       base + slope x tiles on the busiest SM.  256^2: 5.6 us against 8.3 (window), 12.5
//              (streaming), 15.8 (full width); 512^2 9.7 / 13.9 / 19.0 / 19.7.
//   window     2.5 + iterations of the busiest block x time an iteration (choose_rk4_window), times
//              1.12 with a real potential, 1.3 two lasers, 1.7 a complex potential.  600 x 500 x 6
//              with a real potential 31 us against 73 (streaming), 94 (tile); 4096^2 163 against
//              200 (clusters of full-width blocks) and 216 (streaming).
//   full width 1024-site rows, where its bulk copies save a tenth: 8 x 1024^2 71.6 us against
//              82.5 (window); with a real potential the window is ahead (90 against 105).  On narrower
//              rows it is ahead with a complex potential (512^2 x 40: 158 against 183) and, on
//              some grids, with two lasers (512^2 x 4: 24.0 against 25.9).
//   streaming  2.5 + waves x iterations x time an iteration: many small grids (128^2 x 32: 12.3 us
//              against 17.6 for the window, 15.7 for the tile).  Its fit is the loosest: taken 12 %
//              longer, so that it is chosen only where it is clearly ahead.
#include <algorithm>

#include "pg_internal.h"
#include "window_internal.h"

namespace pg {
namespace {

double stream_time(const RK4Geom& g, bool general, bool two, int lasers, int sms) {
  const int threads = g.wrap ? (g.nx + 31) / 32 * 32 : (g.tile_w + 8 + 31) / 32 * 32;
  const int ntx = g.wrap ? 1 : (g.nx + g.tile_w - 1) / g.tile_w;
  const double blocks = static_cast<double>(ntx) * g.members * ((g.ny + g.strip_h - 1) / g.strip_h);
  const int fit = std::max(1, std::min(65536 / (96 * threads), 2048 / threads));
  const int per_sm = std::max(1, std::min(fit, static_cast<int>((blocks + sms - 1) / sms)));
  const double waves = std::max(1.0, blocks / (static_cast<double>(per_sm) * sms));
  const int iters = (g.strip_h + 8 + 3) / 4 * 4;
  const double warps = per_sm * (threads / 32);
  double t = two ? 0.93 + 0.025 * warps : general ? 0.60 + 0.037 * warps : 0.17 + 0.031 * warps;
  if (!g.wrap) t *= 1.2;  // halo columns
  if (lasers > 1) t *= 1.0 + 0.7 * (lasers - 1);  // every envelope read at every stage
  if (static_cast<double>(g.nx) * g.ny * g.members > 3.0e6) t *= 1.25;  // state beyond L2
  return 2.5 + waves * iters * t;
}

// The tile shapes of rk4_tile_f32.cu.
constexpr int kTileW[4] = {16, 16, 32, 32}, kTileH[4] = {8, 16, 16, 32};

long long tile_rows(int shape, int ny) { return (ny + static_cast<long long>(kTileH[shape]) - 1) / kTileH[shape]; }

// Their times, {base, slope} without and with the general right-hand side.
double tile_time(int shape, int nx, int ny, int members, bool general, int sms) {
  static const double fit[4][4] = {{3.4, 0.92, 3.4, 1.95},
                                   {4.2, 1.05, 3.9, 2.75},
                                   {4.0, 1.65, 4.0, 4.2},
                                   {3.3, 3.45, 2.2, 7.5}};
  const double* f = fit[shape];
  const long long tiles = (nx + static_cast<long long>(kTileW[shape]) - 1) / kTileW[shape] * tile_rows(shape, ny) * members;
  const double w = static_cast<double>((tiles + sms - 1) / sms);
  return general ? f[2] + f[3] * w : f[0] + f[1] * w;
}

}  // namespace

namespace {

RK4Route choose_rk4_route(int nx, int ny, int members, int sm_count, const RK4Features& f,
                          const RK4Geom& stream, WindowGeom* window, int* tile) {
  const int sms = sm_count > 0 ? sm_count : 152;
  const bool two = f.reservoir >= 2;
  const bool general = f.potential != 0 || f.relax != 0 || f.reservoir != 1 || f.pump_terms > 1;
  RK4Route route = RK4Route::kStream;
  // The streaming and tile kernels launch a block a member and strip, the others any number of rows
  // on a persistent grid.
  const bool members_fit = members <= kMaxGridYZ;
  double best = 1.12 * stream_time(stream, general, two, f.pump_terms, sms);
  if (!members_fit || (ny + stream.strip_h - 1) / stream.strip_h > kMaxGridYZ) best = 1e300;
  for (int s = 0; s < 4 && members_fit; ++s) {
    if (tile_rows(s, ny) > kMaxGridYZ) continue;
    const double t = tile_time(s, nx, ny, members, general, sms) * (1.0 + 0.2 * (f.pump_terms - 1));
    if (t < best) {
      best = t;
      route = RK4Route::kTile;
      *tile = s;
    }
  }
  if (f.reservoir == 1 && f.pump_terms <= 2) {
    double t = choose_rk4_window(nx, ny, members, sms, window);
    if (t < 0.0) t = 1e300;  // no window fits
    const bool heavy = f.potential == 2;
    t = 2.5 + t * (heavy ? 1.7 : f.pump_terms == 2 ? 1.3 : f.potential ? 1.12 : f.relax ? 1.1 : 1.0);
    if (t < best) {
      best = t;
      route = RK4Route::kWindow;
    }
    if (nx == 1024 || ((heavy || f.pump_terms == 2) && (nx == 128 || nx == 256 || nx == 512))) {
      // whole turns of the 8-row ring
      const long long blocks = row_blocks(members, ny, static_cast<long long>(sms) * (1024 / nx));
      const double iters = (static_cast<int>(row_iterations(members, ny, blocks)) + 7) / 8 * 8;
      const double iter = heavy                 ? 1.78
                          : f.potential == 1    ? 1.64
                          : f.relax             ? 1.41
                          : f.pump_terms == 1   ? 1.13
                          : nx == 1024          ? 1.3
                                                : 1.38;
      t = 2.5 + iters * iter;
      if (t < best) route = RK4Route::kWide;
    }
  }
  return route;
}

}  // namespace

RK4Plan plan_rk4(const pg_config& c, const RK4Features& f, int sm_count) {
  RK4Plan p;
  choose_rk4_geometry(c.nx, c.ny, c.members, c.precision, sm_count, &p.stream);
  if (c.precision == PG_DOUBLE) {
    p.tile = choose_rk4_tile_f64(c.nx, c.ny, c.members, sm_count);
    p.route = p.tile >= 0 ? RK4Route::kTile : RK4Route::kStream;
  } else {
    p.route = choose_rk4_route(c.nx, c.ny, c.members, sm_count, f, p.stream, &p.window, &p.tile);
  }
  return p;
}

}  // namespace pg
