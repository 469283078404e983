// The FP32 split-step passes on the register-resident transforms.
#include "split_reg.cuh"

namespace pg {

cudaError_t configure_split_reg(int nx, int ny) {
  if (reg_fft_size(nx)) {
    const cudaError_t e = configure_row_reg<float>(nx);
    if (e != cudaSuccess) return e;
  }
  return reg_fft_size(ny) ? configure_col_reg<float>(ny) : cudaSuccess;
}

cudaError_t launch_row_reg(float* data, const float* tab, const float* px, const float* py,
                           const RowPassArgs& a, int members, int sm_count,
                           cudaStream_t stream) {
  return launch_row_reg_t<float>(data, tab, px, py, a, members, sm_count, stream);
}

cudaError_t launch_col_reg(float* data, float* res, const float* pump, const float* potential,
                           const float* tab, const SplitConst<float>* consts, const float* scales,
                           const unsigned long long* step_base, const ColPassArgs& a, int sm_count, cudaStream_t stream) {
  return launch_col_reg_t<float>(data, res, pump, potential, tab, consts, scales, step_base, a, sm_count, stream);
}

}  // namespace pg
