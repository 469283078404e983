// Which kernel steps a grid when the caller leaves the choice.  FP64: the tile kernel (rk4_tile_f64.cu;
// measured without / with Wigner noise, us a step, streaming kernel -> tile kernel: 92.6 -> 11.4 /
// 141 -> 14.7 at 128^2, 179 -> 24.4 / 269 -> 35.9 at 256^2, 208 -> 78 / 314 -> 123 at 512^2,
// 310 -> 268 / 495 -> 426 at 1024^2), where its launch fits.  FP32: the tile kernel (rk4_tile.cuh),
// the window kernel (rk4_window.cuh), the full-width kernel (rk4_wide.cu) or the streaming kernel
// (rk4.cu).  All give the same bits, so the choice is the smallest modelled time.
//
// The models (us a step) are fitted to 17000 measurements on 198 grids from 48 x 50 to 4096^2 in one to
// 1591 members, with and without Wigner noise, to 3-8 % rms each.  An SM's four schedulers set the time of an
// iteration of the row kernels: it depends on the warps resident on the busiest SM in steps of four,
// and on the right-hand side.  Without noise, with it:
//   tile       256^2 5.2 / 5.6 us against 6.8 / 8.2 (window), 9.8 / 12.1 (streaming), 9.4 / 11.5 (full width)
//   window     600 x 500 x 6 with a real potential 25 / 31 us against 62 / 71 (streaming), 87 / 94 (tile);
//              4096^2 107 / 164 against 157 / 202 (full width, clusters), 165 / 211 (streaming)
//   full width 1024^2 x 8 52 / 74 us against 58 / 82 (window); with a real potential 94 / 107 against 70 / 93
//   streaming  64^2 x 64 7.9 / 9.7 us against 9.5 / 12.4 (window), 8.7 / 9.7 (tile)
// Which is ahead can change with the noise (64^2 x 64), so the choice is made again when it is turned on or off.
#include <algorithm>
#include <cmath>

#include "pg_internal.h"
#include "wide_internal.h"
#include "window_internal.h"

namespace pg {
namespace {

// Kinds of right-hand side, by what they cost.
enum Kind { kPlain, kRelax, kReal, kComplex, kLasers, kTwo, kNone, kKinds };

Kind kind_of(const RK4Features& f) {
  if (f.reservoir == 0) return kNone;
  if (f.reservoir >= 2) return kTwo;
  if (f.pump_terms > 1) return kLasers;
  if (f.potential) return f.potential == 2 ? kComplex : kReal;
  return f.relax ? kRelax : kPlain;
}

// Warps of the busiest SM in units of its four schedulers, 0-based, at most `most`.
int load(long long warps, int most) {
  return static_cast<int>(std::min<long long>(most, std::max<long long>(1, (warps + 3) / 4))) - 1;
}

// States beyond some 110 MB, of the 129 MB level-2 cache, stream from memory.
bool beyond_l2(int nx, int ny, int members) { return static_cast<double>(nx) * ny * members > 4.0e6; }

// Microseconds of a launch and of an iteration with at most four warps an SM by kind, without and with noise,
// and what the iteration takes more with up to 8, 12, 16 and 20.
constexpr double kStreamIter[2][kKinds] = {{0.203, 0.675, 0.824, 0.839, 1.547, 0.972, 0.620},
                                           {0.341, 0.714, 0.850, 0.863, 1.566, 1.055, 0.670}};
constexpr double kStreamLoad[2][2][5] = {{{0.0, 0.068, 0.177, 0.285, 0.369}, {0.0, 0.094, 0.234, 0.374, 0.506}},
                                         {{0.0, 0.047, 0.127, 0.238, 0.344}, {0.0, 0.066, 0.179, 0.336, 0.485}}};
double stream_time(const RK4Geom& g, Kind kind, int lasers, bool noise, int sms) {
  const int warps = (g.wrap ? g.nx + 31 : g.tile_w + 8 + 31) / 32;
  const int ntx = g.wrap ? 1 : (g.nx + g.tile_w - 1) / g.tile_w;
  const long long blocks = static_cast<long long>(ntx) * g.members * ((g.ny + g.strip_h - 1) / g.strip_h);
  // 96 registers a thread: five warps a scheduler.
  const long long per_sm = std::min<long long>(std::max(1, 20 / warps), (blocks + sms - 1) / sms);
  double waves = static_cast<double>(blocks) / static_cast<double>(per_sm * sms);
  waves = waves < 4.0 ? std::ceil(waves) : waves + 0.3;
  const int iters = (g.strip_h + 8 + 3) / 4 * 4;
  double t = kStreamIter[noise][kind] + kStreamLoad[kind != kPlain][noise][load(per_sm * warps, 5)];
  if (lasers > 2) t += 0.74 * (lasers - 2);  // every envelope read at every stage
  if (beyond_l2(g.nx, g.ny, g.members)) t *= 1.16;
  return (kind != kPlain ? 1.0 : noise ? 1.7 : 3.3) + waves * iters * t;
}

// The tile shapes of rk4_tile_f32.cu.
constexpr int kTileW[4] = {16, 16, 32, 32}, kTileH[4] = {8, 16, 16, 32};

long long tile_rows(int shape, int ny) { return (ny + static_cast<long long>(kTileH[shape]) - 1) / kTileH[shape]; }

// Microseconds for a further 16 x 8 tile on the busiest SM; the times of one tile and of more of each
// shape are linear in it.
constexpr double kTileMore[2][kKinds] = {{0.0, 1.530, 1.969, 1.988, 2.347, 1.688, 1.385},
                                         {0.0, 1.645, 2.085, 2.102, 2.463, 1.806, 1.500}};
// The plain right-hand side: one tile, and more as a constant and a slope.
constexpr double kTilePlain[2][4][3] = {
    {{3.97, 2.98, 0.736}, {4.58, 3.04, 1.023}, {5.48, 3.30, 1.523}, {6.25, 2.34, 3.109}},
    {{4.19, 2.74, 0.957}, {4.88, 3.09, 1.134}, {5.95, 3.28, 1.776}, {6.76, 2.28, 3.586}}};
double tile_time(int shape, int nx, int ny, int members, Kind kind, int lasers, bool noise, int sms) {
  static const double fit[4][5] = {{2.02, 1.74, 3.13, -0.61, 1.0},
                                   {1.38, 2.68, 1.80, -0.10, 1.443},
                                   {1.00, 3.92, 0.02, 0.64, 2.175},
                                   {1.43, 3.81, 1.04, -0.83, 4.082}};
  const long long tiles = (nx + static_cast<long long>(kTileW[shape]) - 1) / kTileW[shape] * tile_rows(shape, ny) * members;
  const long long w = (tiles + sms - 1) / sms;
  if (kind == kPlain) {
    const double* p = kTilePlain[noise][shape];
    return w == 1 ? p[0] : p[1] + p[2] * static_cast<double>(w);
  }
  const double* f = fit[shape];
  const double more = kTileMore[noise][kind] + (lasers > 2 ? 0.44 * (lasers - 2) : 0.0);
  return w == 1 ? f[0] + f[1] * more : f[2] + (f[3] + f[4] * static_cast<double>(w)) * more;
}

// Microseconds an iteration with one to four warps a scheduler, by kind, without and with noise.
constexpr double kWindowIter[2][5][4] = {{{0.413, 0.459, 0.641, 0.814},
                                          {0.656, 0.648, 0.812, 0.992},
                                          {0.680, 0.671, 0.843, 1.038},
                                          {1.061, 1.261, 1.414, 1.618},
                                          {0.853, 0.860, 1.005, 1.294}},
                                         {{0.690, 0.740, 0.967, 1.207},
                                          {0.727, 0.806, 1.114, 1.407},
                                          {0.758, 0.827, 1.116, 1.412},
                                          {1.143, 1.354, 1.582, 1.930},
                                          {0.987, 1.067, 1.211, 1.631}}};
// Iterations that a block loses where it crosses from one member or band into the next, beyond the 8
// of fill: a new set of constants and an empty ring.
constexpr double kWindowCross[2][5] = {{0.5, 0.0, 0.0, 18.3, 18.3}, {5.3, 26.0, 26.0, 38.3, 38.3}};
double window_time(const WindowGeom& g, Kind kind, bool noise, int sms) {
  const int w = g.bands == 1 ? g.nx : g.band_w + 8;
  const int warps = ((w + 1) / 2 + 31) / 32;
  const long long units = static_cast<long long>(g.members) * g.bands;
  double iters;
  if (g.blocks % units == 0)
    iters = (g.ny + g.blocks / units - 1) / (g.blocks / units) + 8.0;
  else
    iters = static_cast<double>((units * g.ny + g.blocks - 1) / g.blocks) + 8.0 +
            (8.0 + kWindowCross[noise][kind]) * static_cast<double>(units) / g.blocks;
  double t = kWindowIter[noise][kind][load(warps * ((g.blocks + static_cast<long long>(sms) - 1) / sms), 4)];
  if (beyond_l2(g.nx, g.ny, g.members)) t *= 1.10;
  if (g.nx % 2) t *= 1.05;  // copies of single elements
  return (kind != kPlain ? 1.0 : noise ? 1.2 : 2.7) + iters * t;
}

constexpr double kWideIter[2][5][4] = {{{0.286, 0.394, 0.514, 0.700},
                                        {0.534, 0.599, 0.794, 0.940},
                                        {0.721, 0.846, 1.004, 1.199},
                                        {0.785, 1.005, 1.112, 1.377},
                                        {0.578, 0.645, 0.842, 1.036}},
                                       {{0.422, 0.564, 0.756, 1.009},
                                        {0.571, 0.676, 0.935, 1.228},
                                        {0.687, 0.874, 1.063, 1.388},
                                        {0.754, 1.013, 1.146, 1.507},
                                        {0.614, 0.717, 0.980, 1.276}}};
double wide_time(int nx, int ny, int members, Kind kind, bool noise, int sms) {
  const int size = std::max(1, nx / 1024);  // CTAs of a cluster
  long long streams, warps = 16;            // row streams
  if (size > 1) {
    streams = std::max<long long>(1, std::min<long long>(size == 2 ? sms / 2 : sms / size - 2,
                                                         static_cast<long long>(members) * ny / 16));
  } else {
    streams = wide_rk4_blocks(nx, ny, members, 1024 / nx, sms);
    warps = (streams + sms - 1) / sms * nx / 64;
  }
  long long iters;
  if (streams % members == 0) {
    iters = (ny + streams / members - 1) / (streams / members) + 8;
  } else {
    const long long rows = (static_cast<long long>(members) * ny + streams - 1) / streams;
    iters = rows + 8 * (2 + std::max<long long>(0, rows - 2) / ny);
  }
  double t = kWideIter[noise][kind][load(warps, 4)];
  const bool heavy = kind == kReal || kind == kComplex;
  if (size > 1)
    t *= 1.43;  // edges from the neighbouring CTA
  else if (nx == 1024)
    t *= heavy ? 0.99 : 0.849;  // bulk copies of whole rows
  else if (nx == 256)
    t *= noise ? 1.096 : 1.071;
  else if (nx == 128)
    t *= noise ? 1.191 : 1.128;
  if (beyond_l2(nx, ny, members)) t *= 1.18;
  return 4.5 + static_cast<double>((iters + 7) / 8 * 8) * t;  // whole turns of the 8-row ring
}

// Kernels other than the streaming one, or the full-width one where it takes the grid, have to be this much
// ahead: the models are no better.
constexpr double kMargin = 1.03;

RK4Route choose_rk4_route(int nx, int ny, int members, int sm_count, const RK4Features& f, bool noise,
                          const RK4Geom& stream, WindowGeom* window, int* tile) {
  const int sms = sm_count > 0 ? sm_count : 152;
  const Kind kind = kind_of(f);
  const bool row_kernels = f.reservoir == 1 && f.pump_terms <= 2;
  const bool wide = row_kernels && wide_rk4_supported(nx, ny) && nx <= (f.pump_terms == 1 ? 8192 : 1024);
  // The streaming and tile kernels launch a block a member and strip, the others any number of rows
  // on a persistent grid.
  const bool members_fit = members <= kMaxGridYZ;
  RK4Route route = RK4Route::kStream;
  double best = stream_time(stream, kind, f.pump_terms, noise, sms) * (wide ? kMargin : 1.0);
  if (!members_fit || (ny + stream.strip_h - 1) / stream.strip_h > kMaxGridYZ) best = 1e300;
  auto take = [&](double t, RK4Route r) {
    if (t >= best) return false;
    best = t;
    route = r;
    return true;
  };
  if (wide) take(wide_time(nx, ny, members, kind, noise, sms), RK4Route::kWide);
  for (int s = 0; s < 4 && members_fit; ++s)
    if (tile_rows(s, ny) <= kMaxGridYZ &&
        take(kMargin * tile_time(s, nx, ny, members, kind, f.pump_terms, noise, sms), RK4Route::kTile))
      *tile = s;
  if (row_kernels && choose_rk4_window(nx, ny, members, sms, window))
    take(kMargin * window_time(*window, kind, noise, sms), RK4Route::kWindow);
  return route;
}

}  // namespace

RK4Plan plan_rk4(const pg_config& c, const RK4Features& f, bool noise, int sm_count) {
  RK4Plan p;
  choose_rk4_geometry(c.nx, c.ny, c.members, c.precision, sm_count, &p.stream);
  if (c.precision == PG_DOUBLE) {
    p.tile = choose_rk4_tile_f64(c.nx, c.ny, c.members, sm_count);
    p.route = p.tile >= 0 ? RK4Route::kTile : RK4Route::kStream;
  } else {
    p.route = choose_rk4_route(c.nx, c.ny, c.members, sm_count, f, noise, p.stream, &p.window, &p.tile);
  }
  return p;
}

}  // namespace pg
