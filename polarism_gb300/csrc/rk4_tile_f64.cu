// The FP64 tile shapes of the RK4 tile kernel (rk4_tile.cuh) and the rule that picks one.
//
// What bounds it: the FP64 pipe.  A GB300 SM retires two FP64 lanes a clock, so a warp's FP64
// instruction holds the pipe for 16 cycles, and a site-stage is about 26 of them; everything else
// (shared memory, index arithmetic) hides behind it.  A step's time is therefore the site-stages
// of the busiest SM.  The streaming kernel gave a 128^2 grid 8 blocks of 24 rows each -- 8 SMs of
// 152; 16 x 8 tiles give it 128 SMs (92.6 -> 11.4 us a step; FP64 pipe floor of the useful work on
// all SMs 2.9 us, of these tiles 5.7).
#include "rk4_tile.cuh"

namespace pg {

// The tile whose busiest SM has the fewest 32-site units: tiles per SM, rounded up, times the
// units of a tile.  Small tiles spread a small grid over the SMs, large ones recompute less: us a
// step for 16 x 8 / 16 x 16 / 32 x 16 / 32 x 32 tiles (no noise) 11.4 / 16.0 / 24.2 / 40.2 at
// 128^2, 33.1 / 27.0 / 24.4 / 40.5 at 256^2, 106 / 82 / 81 / 78 at 512^2, 396 / 303 / 272 / 268 at
// 1024^2; the rule takes the fastest in each.  -1: no launch holds the grid (its y and z dimensions count
// tile rows and members).
int choose_rk4_tile_f64(int nx, int ny, int members, int sm_count) {
  const long long sms = sm_count > 0 ? sm_count : 152;
  struct Shape { int w, h, units; };
  const Shape shapes[] = {{16, 8, TileShape<16, 8>::units()},
                          {16, 16, TileShape<16, 16>::units()},
                          {32, 16, TileShape<32, 16>::units()},
                          {32, 32, TileShape<32, 32>::units()}};
  int best = -1;
  long long best_cost = -1;
  if (members > kMaxGridYZ) return best;
  for (int i = 0; i < 4; ++i) {
    if ((ny + static_cast<long long>(shapes[i].h) - 1) / shapes[i].h > kMaxGridYZ) continue;
    const long long tiles = static_cast<long long>((nx + shapes[i].w - 1) / shapes[i].w) *
                            ((ny + shapes[i].h - 1) / shapes[i].h) * members;
    const long long cost = (tiles + sms - 1) / sms * shapes[i].units;
    if (best_cost < 0 || cost < best_cost) {
      best = i;
      best_cost = cost;
    }
  }
  return best;
}

cudaError_t launch_rk4_tile_f64(int shape, const double* psi_in, const double* n_in, const double* pump,
                                const double* potential, double* psi_out, double* n_out,
                                const RhsConst<double>* consts, const double* scales,
                                const unsigned long long* step_base, int step_offset, double dt,
                                bool noise, const RK4Geom& g, const RK4Features& f,
                                cudaStream_t stream) {
  switch (shape) {
#define PG_TILE_CASE(I, W, H, WARPS, MINB)                                                         \
  case I:                                                                                          \
    return launch_tile_shape<double, W, H, WARPS, MINB>(psi_in, n_in, pump, potential, psi_out,    \
                                                        n_out, consts, scales, step_base,          \
                                                        step_offset, dt, noise, g, f, stream);
    PG_TILE_CASE(0, 16, 8, 10, 2)
    PG_TILE_CASE(1, 16, 16, 8, 2)
    PG_TILE_CASE(2, 32, 16, 8, 2)
    PG_TILE_CASE(3, 32, 32, 16, 1)
#undef PG_TILE_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace pg
