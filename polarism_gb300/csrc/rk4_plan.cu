// Which kernel steps a grid when the caller leaves the choice.  FP64: the tile kernel (rk4_tile_f64.cu;
// measured without / with Wigner noise, us a step, streaming kernel -> tile kernel: 92.6 -> 11.4 /
// 141 -> 14.7 at 128^2, 179 -> 24.4 / 269 -> 35.9 at 256^2, 208 -> 78 / 314 -> 123 at 512^2,
// 310 -> 268 / 495 -> 426 at 1024^2), where its launch fits.  FP32: the tile kernel (rk4_tile.cuh),
// the window kernel (rk4_window.cuh), the full-width kernel (rk4_wide.cu) or the streaming kernel
// (rk4.cu).  All give the same bits, so the choice is the smallest modelled time.
//
// The models (us a step) are fitted to 26000 measurements on 640 grids from 48 x 50 to 4096^2 in one to
// 1591 members, with and without Wigner noise, to 2-7 % rms each; on 735 cases of 220 other grids the choice
// is 0.1 % slower than the fastest kernel in the mean, and more than 5 % in 7.  An SM's four schedulers set the
// time of an iteration of the row kernels: it depends on the warps resident on the busiest SM in steps of
// four, and on the right-hand side.  Without noise, with it:
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

// Microseconds of an iteration with at most four warps an SM by kind, without and with noise, and what it takes
// more with up to 8, 12, 16 and 20 (plain, the other kinds, a potential or lasers) and where the row ends inside a warp; the factor of
// states that stream from memory.
constexpr double kStreamIter[2][kKinds] = {{0.201, 0.675, 0.786, 0.800, 1.531, 0.963, 0.632},
                                           {0.333, 0.710, 0.824, 0.838, 1.570, 1.038, 0.680}};
constexpr double kStreamLoad[3][2][5] = {{{0.0, 0.065, 0.145, 0.285, 0.381}, {0.0, 0.091, 0.208, 0.362, 0.501}},
                                         {{0.0, 0.048, 0.120, 0.217, 0.308}, {0.0, 0.075, 0.176, 0.315, 0.447}},
                                         {{0.0, 0.056, 0.141, 0.272, 0.408}, {0.0, 0.080, 0.186, 0.357, 0.521}}};
constexpr double kStreamRagged[2][2] = {{0.035, 0.032}, {0.014, 0.014}};
constexpr double kStreamBig[kKinds] = {1.15, 1.20, 1.17, 1.17, 1.06, 1.30, 1.14};
double stream_time(const RK4Geom& g, Kind kind, int lasers, bool noise, int sms) {
  const int warps = (g.wrap ? g.nx + 31 : g.tile_w + 8 + 31) / 32;
  const int ntx = g.wrap ? 1 : (g.nx + g.tile_w - 1) / g.tile_w;
  const long long blocks = static_cast<long long>(ntx) * g.members * ((g.ny + g.strip_h - 1) / g.strip_h);
  // 96 registers a thread: five warps a scheduler.
  const long long per_sm = std::min<long long>(std::max(1, 20 / warps), (blocks + sms - 1) / sms);
  const long long slots = per_sm * sms;
  const int iters = (g.strip_h + 8 + 3) / 4 * 4;
  const bool general = kind != kPlain;
  double base = kStreamIter[noise][kind] + (g.wrap && g.nx % 32 ? kStreamRagged[general][noise] : 0.0);
  if (lasers > 2) base += 0.74 * (lasers - 2);  // every envelope read at every stage
  const int group = kind == kPlain ? 0 : kind == kReal || kind == kComplex || kind == kLasers ? 2 : 1;
  auto wave = [&](long long w) { return base + kStreamLoad[group][noise][load(w, 5)]; };
  double t = wave(per_sm * warps);
  if (blocks >= 4 * slots) {
    t *= static_cast<double>(blocks) / static_cast<double>(slots) + 0.3;
  } else if (blocks > slots) {
    // whole waves, and a last one with what is left on each SM
    const long long left = blocks % slots;
    t *= static_cast<double>(blocks / slots);
    if (left) t += wave((left + sms - 1) / sms * warps);
  }
  if (beyond_l2(g.nx, g.ny, g.members)) t *= kStreamBig[kind];
  if (!g.wrap) t *= 1.012;
  return (general ? 1.0 : noise ? 1.7 : 3.2) + iters * t;
}

// The tile shapes of rk4_tile_f32.cu.
constexpr int kTileW[4] = {16, 16, 32, 32}, kTileH[4] = {8, 16, 16, 32};

long long tile_rows(int shape, int ny) { return (ny + static_cast<long long>(kTileH[shape]) - 1) / kTileH[shape]; }

// Tiles of each shape that an SM holds at once, plain and other right-hand sides: a further round of them costs
// a step in the time (real potential and noise: 9.5, 10.5, 18.5 and 18.8 us with one to four 32 x 16 tiles an SM).
constexpr int kTileRound[2][4] = {{3, 4, 4, 2}, {2, 2, 2, 1}};
// Microseconds of one tile, of a further round and of a further tile in a round with the plain right-hand side.
constexpr double kTilePlain[2][4][3] = {
    {{3.92, 2.17, 0.68}, {4.63, 3.92, 0.77}, {5.50, 5.80, 1.23}, {6.36, 5.82, 2.35}},
    {{4.21, 2.82, 0.58}, {4.89, 4.41, 0.80}, {5.94, 6.85, 1.36}, {6.86, 6.79, 2.70}}};
// The other kinds: microseconds for a further round of 16 x 8 tiles, and in its terms a constant, the slopes
// of one tile, of a round and of a further tile in one for each shape.
constexpr double kTileMore[2][kKinds] = {{0.0, 2.896, 3.744, 3.780, 4.506, 3.187, 2.677},
                                         {0.0, 3.108, 3.980, 4.017, 4.718, 3.406, 2.870}};
constexpr double kTileShape[4][4] = {{2.459, 0.803, 1.000, 0.135},
                                     {1.535, 1.375, 1.413, 0.191},
                                     {0.000, 2.357, 2.094, 0.274},
                                     {1.337, 2.028, 1.954, 0.0}};
constexpr double kTileBig[kKinds] = {1.06, 1.15, 1.13, 1.13, 1.13, 1.15, 1.09};
double tile_time(int shape, int nx, int ny, int members, Kind kind, int lasers, bool noise, int sms) {
  const long long tiles = (nx + static_cast<long long>(kTileW[shape]) - 1) / kTileW[shape] * tile_rows(shape, ny) * members;
  const long long w = (tiles + sms - 1) / sms, held = kTileRound[kind != kPlain][shape];
  const double rounds = static_cast<double>((w - 1) / held), further = static_cast<double>((w - 1) % held);
  const bool big = beyond_l2(nx, ny, members);
  if (kind == kPlain) {
    const double* p = kTilePlain[noise][shape];
    return (p[0] + p[1] * rounds + p[2] * further) * (big ? kTileBig[kind] : 1.0);
  }
  const double* f = kTileShape[shape];
  const double more = kTileMore[noise][kind] + (lasers > 2 ? 0.88 * (lasers - 2) : 0.0);
  return (f[0] + more * (f[1] + f[2] * rounds + f[3] * further)) * (big ? kTileBig[kind] : 1.0);
}

// Microseconds an iteration with one to four warps a scheduler, by kind, without and with noise.
constexpr double kWindowIter[2][5][4] = {{{0.420, 0.480, 0.663, 0.832},
                                          {0.647, 0.658, 0.830, 1.008},
                                          {0.673, 0.683, 0.861, 1.039},
                                          {1.053, 1.276, 1.427, 1.556},
                                          {0.843, 0.872, 1.018, 1.271}},
                                         {{0.691, 0.758, 0.990, 1.241},
                                          {0.716, 0.818, 1.135, 1.410},
                                          {0.750, 0.834, 1.118, 1.395},
                                          {1.138, 1.371, 1.613, 1.877},
                                          {0.976, 1.085, 1.226, 1.596}}};
// The same relative to its class by the warps on an SM: blocks of an odd number of warps load the schedulers
// unevenly, most with three blocks of five.
constexpr double kWindowWarps[16] = {1.0,   1.0,   1.0, 1.0, 0.968, 0.954, 1.009, 1.0,
                                     0.926, 0.963, 1.0, 1.0, 1.0,   0.950, 1.041, 1.0};
constexpr double kWindowBig[5] = {1.06, 1.07, 1.08, 1.18, 1.12};
// Iterations that a block loses where it crosses from one member or band into the next, beyond the 8
// of fill: a new set of constants and an empty ring.
constexpr double kWindowCross[2][5] = {{0.5, 0.1, 0.1, 18.2, 18.2}, {5.3, 26.0, 26.0, 38.2, 38.2}};
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
  const long long resident = std::min<long long>(16, warps * ((g.blocks + static_cast<long long>(sms) - 1) / sms));
  double t = kWindowIter[noise][kind][load(resident, 4)] * kWindowWarps[resident - 1];
  if (beyond_l2(g.nx, g.ny, g.members)) t *= kWindowBig[kind];
  if (g.nx % 2) t *= 1.048;  // copies of single elements
  return (kind != kPlain ? 1.1 : noise ? 1.2 : 2.7) + iters * t;
}

// The same for rows of up to 512 sites, of 1024 (bulk copies of whole rows; always 16 warps) and for a CTA of a
// cluster (edges from the neighbouring CTA; one laser).
constexpr double kWideIter[2][5][4] = {{{0.273, 0.388, 0.502, 0.670},
                                        {0.519, 0.590, 0.777, 0.970},
                                        {0.733, 0.852, 1.027, 1.223},
                                        {0.794, 1.008, 1.144, 1.392},
                                        {0.563, 0.636, 0.825, 1.060}},
                                       {{0.405, 0.558, 0.739, 1.007},
                                        {0.555, 0.666, 0.915, 1.225},
                                        {0.721, 0.883, 1.120, 1.419},
                                        {0.789, 1.028, 1.211, 1.552},
                                        {0.598, 0.707, 0.959, 1.296}}};
constexpr double kWide1024[2][5] = {{0.735, 0.903, 1.317, 1.566, 0.954}, {1.075, 1.145, 1.470, 1.619, 1.176}};
constexpr double kWideCluster[2][4] = {{1.028, 1.149, 1.598, 1.813}, {1.227, 1.666, 1.977, 2.094}};
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
  const double turns = static_cast<double>((iters + 7) / 8 * 8);  // of the 8-row ring, in iterations
  const bool big = beyond_l2(nx, ny, members);
  if (size > 1) return 8.5 + turns * kWideCluster[noise][kind] * (big ? 1.22 : 1.0) * (size == 3 ? 1.02 : 1.0);
  if (nx == 1024) return 2.5 + turns * kWide1024[noise][kind] * (big ? 1.07 : 1.0);
  double t = kWideIter[noise][kind][load(warps, 4)];
  const bool heavy = kind == kReal || kind == kComplex;
  if (nx == 256)
    t *= heavy ? 1.06 : noise ? 1.114 : 1.079;
  else if (nx == 128)
    t *= heavy ? (noise ? 1.115 : 1.089) : noise ? 1.215 : 1.152;
  return 4.6 + turns * t * (big ? 1.17 : 1.0);
}

// Kernels other than the streaming one, or the full-width one where it takes the grid, have to be this much
// ahead: the models are no better, least with two reservoir fields.
constexpr double margin_of(Kind kind) { return kind == kTwo ? 1.05 : 1.015; }

RK4Route choose_rk4_route(int nx, int ny, int members, int sm_count, const RK4Features& f, bool noise,
                          const RK4Geom& stream, WindowGeom* window, int* tile) {
  const int sms = sm_count > 0 ? sm_count : 152;
  const Kind kind = kind_of(f);
  const double margin = margin_of(kind);
  const bool row_kernels = f.reservoir == 1 && f.pump_terms <= 2;
  const bool wide = row_kernels && wide_rk4_supported(nx, ny) && nx <= (f.pump_terms == 1 ? 8192 : 1024);
  // The streaming and tile kernels launch a block a member and strip, the others any number of rows
  // on a persistent grid.
  const bool members_fit = members <= kMaxGridYZ;
  RK4Route route = RK4Route::kStream;
  double best = stream_time(stream, kind, f.pump_terms, noise, sms) * (wide ? margin : 1.0);
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
        take(margin * tile_time(s, nx, ny, members, kind, f.pump_terms, noise, sms), RK4Route::kTile))
      *tile = s;
  if (row_kernels && choose_rk4_window(nx, ny, members, sms, window))
    take(margin * window_time(*window, kind, noise, sms), RK4Route::kWindow);
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
