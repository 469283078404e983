// Internal declarations of the FP32 RK4 window kernel (rk4_window.cuh).
#pragma once
#include <cuda_runtime.h>

#include "pg_internal.h"

namespace pg {

struct WindowGeom {
  int nx, ny, members;
  int bands;               // windows a row; 1: the row closes on itself
  int band_w;              // columns a band writes (even when bands > 1)
  int wmax;                // window capacity: 256, 320, 512 or 1024 columns
  int blocks;              // persistent grid
  long long pump_stride;   // 0: shared envelope; nx*ny: one per member
  int pump_terms;
  long long pump_term_stride;
  const int* halt;
  const float* pot;        // potential: none, real or complex (pot_kind 0, 1, 2)
  long long pot_stride;
  int pot_kind;
  int relax;
  int wait_limit;          // polls of a wait on the split barrier, before it gives up
};

// The kernel a grid is stepped with when the caller leaves the choice, and the geometry of each
// (rk4_plan.cu).
struct RK4Plan {
  RK4Route route = RK4Route::kStream;
  RK4Geom stream{};
  WindowGeom window{};  // FP32
  int tile = 0;         // tile shape of rk4_tile_f32.cu / rk4_tile_f64.cu
};
RK4Plan plan_rk4(const pg_config& cfg, const RK4Features& f, bool noise, int sm_count);

double row_iterations(long long units, int ny, long long blocks);
long long row_blocks(long long units, int ny, long long slots);
// Picks bands, band_w, wmax and blocks for a grid; false if no window holds it (rows beyond some 500,000
// sites).
bool choose_rk4_window(int nx, int ny, int members, int sm_count, WindowGeom* g);
cudaError_t launch_rk4_window(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                              float* n_out, const RhsConst<float>* consts, const float* scales,
                              const unsigned long long* step_base, int step_offset, float dt, bool noise,
                              const WindowGeom& g, int* err_flag, cudaStream_t stream);
// The same for one window capacity, instantiated in the rk4_window_<capacity>.cu (one each, to compile in
// parallel).
template <int WMAX>
cudaError_t launch_window_t(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                            float* n_out, const RhsConst<float>* consts, const float* scales,
                            const unsigned long long* step_base, int step_offset, float dt, bool noise,
                            const WindowGeom& g, int* err_flag, cudaStream_t stream);

}  // namespace pg
