// Launch geometry of the FP32 RK4 window kernel (rk4_window.cuh).
#include <algorithm>

#include "window_internal.h"

namespace pg {

// Iterations of the busiest block when `units` columns of `ny` rows go to `blocks` blocks: its rows
// plus the 8 rows of fill, once more where a block crosses from one unit into the next.
double row_iterations(long long units, int ny, long long blocks) {
  if (blocks % units == 0) return (ny + blocks / units - 1) / (blocks / units) + 8.0;
  return static_cast<double>((units * ny + blocks - 1) / blocks) + 16.0;
}

// The block count of at most `slots`: whole strips of units where the busiest block then has clearly
// fewer iterations (a few per cent less on it alone is lost on the SMs left without a block).
long long row_blocks(long long units, int ny, long long slots) {
  const long long rows = units * ny;
  long long best = std::min(slots, rows);
  if (units <= slots) {
    const long long strips = units * std::min<long long>(slots / units, ny);
    if (row_iterations(units, ny, strips) <= 0.95 * row_iterations(units, ny, best)) best = strips;
  }
  return best;
}

// The window and the grid whose modelled time is smallest.  A block advances h rows in h + 8
// iterations; an iteration of an SM with W resident warps takes max(0.68, 0.36 + 0.056 W) us: the
// dependency chain of one thread, or issue slots (measured with Wigner noise on grids from 256^2
// to 4096^2, windows of 3 to 16 warps, one to four blocks an SM: 0.66-0.73 us with 3 to 6 warps,
// 0.79-0.97 with 8 to 10, 1.02-1.1 with 12, 1.2-1.3 with 16).  False where no window of these capacities takes the row.
bool choose_rk4_window(int nx, int ny, int members, int sm_count, WindowGeom* g) {
  const int sms = sm_count > 0 ? sm_count : 152;
  const int capacity[] = {256, 320, 512, 1024};
  double best = -1.0;
  for (int wmax : capacity) {
    const int fit = 512 / (wmax / 2);  // blocks an SM
    for (int bands = 1; bands <= nx; ++bands) {
      int band_w = nx, w = nx + (nx & 1);
      if (bands > 1) {
        if (nx < 32) break;  // a window never wraps more than once around the row
        band_w = (nx + bands - 1) / bands;
        band_w += band_w & 1;
        w = band_w + 8;
        if (static_cast<long long>(band_w) * (bands - 1) >= nx) break;  // an empty last band
      }
      if (w > wmax) continue;
      const int warps = ((w + 1) / 2 + 31) / 32;
      const long long units = static_cast<long long>(members) * bands;
      for (int per_sm = 1; per_sm <= fit; ++per_sm) {
        const long long blocks = row_blocks(units, ny, static_cast<long long>(per_sm) * sms);
        // one block an SM (the split barrier) is 8 % slower an iteration than its warps alone say
        const double cost = row_iterations(units, ny, blocks) * (wmax > 512 ? 1.08 : 1.0) *
                            std::max(0.68, 0.36 + 0.056 * per_sm * warps);
        if (best < 0.0 || cost < best * 0.999) {
          best = cost;
          g->bands = bands;
          g->band_w = band_w;
          g->wmax = wmax;
          g->blocks = static_cast<int>(blocks);
        }
      }
      if (bands > 1 && band_w + 8 <= wmax / 2) break;  // narrower windows only recompute more
    }
  }
  g->nx = nx;
  g->ny = ny;
  g->members = members;
  return best >= 0.0;
}

cudaError_t launch_rk4_window(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                              float* n_out, const RhsConst<float>* consts, const float* scales,
                              const unsigned long long* step_base, int step_offset, float dt, bool noise,
                              const WindowGeom& g, int* err_flag, cudaStream_t stream) {
  switch (g.wmax) {
#define PG_WIN_CASE(W)                                                                                  \
  case W:                                                                                               \
    return launch_window_t<W>(psi_in, n_in, pump, psi_out, n_out, consts, scales, step_base,            \
                              step_offset, dt, noise, g, err_flag, stream);
    PG_WIN_CASE(256)
    PG_WIN_CASE(320)
    PG_WIN_CASE(512)
    PG_WIN_CASE(1024)
#undef PG_WIN_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace pg
