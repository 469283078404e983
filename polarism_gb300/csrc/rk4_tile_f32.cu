// The FP32 tile shapes of the RK4 tile kernel (rk4_tile.cuh; rk4_plan.cu picks one).
//
// On small grids a step is latency: the row kernels walk at least 16 rows one after another, a tile
// makes four dependent stages however large the grid.  One 256^2 member: 5.6 us a step against 12.5
// (streaming kernel) and 15.8 (full-width kernel).
#include "rk4_tile.cuh"

namespace pg {

cudaError_t launch_rk4_tile_f32(int shape, const float* psi_in, const float* n_in, const float* pump,
                                const float* potential, float* psi_out, float* n_out,
                                const RhsConst<float>* consts, const float* scales,
                                const unsigned long long* step_base, int step_offset, float dt,
                                bool noise, const RK4Geom& g, const RK4Features& f,
                                cudaStream_t stream) {
  switch (shape) {
#define PG_TILE_CASE(I, W, H, WARPS, MINB)                                                         \
  case I:                                                                                          \
    return launch_tile_shape<float, W, H, WARPS, MINB>(psi_in, n_in, pump, potential, psi_out,    \
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
