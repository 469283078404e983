// The RK4 window kernel for windows of at most 256 columns.
#include "rk4_window.cuh"

namespace pg {

cudaError_t launch_rk4_window_256(const float* psi_in, const float* n_in, const float* pump, float* psi_out,
                                 float* n_out, const RhsConst<float>* consts, const float* scales,
                                 const unsigned long long* step_base, int step_offset, float dt, bool noise,
                                 const WindowGeom& g, int* err_flag, cudaStream_t stream) {
  return launch_window_t<256>(psi_in, n_in, pump, psi_out, n_out, consts, scales, step_base, step_offset, dt,
                             noise, g, err_flag, stream);
}

}  // namespace pg
