// Internal declarations of the split-step (Stockham FFT) passes.
#pragma once
#include <cuda_runtime.h>

namespace pg {

enum SplitOp {
  SPLIT_OP_NONE = 0,
  SPLIT_OP_KOUTER = 1,         // R(dt/2) at P(t+dt/4), N(dt), R(dt/2) at P(t+3dt/4), Wigner
  SPLIT_OP_RES_START = 2,      // R(dt/2) at P(t+dt/4)
  SPLIT_OP_RES_END_START = 3,  // R(dt/2) at P(t-dt/4) of the previous step, then at P(t+dt/4)
  SPLIT_OP_NONLINEAR = 4,      // N(dt), then Wigner with the current n_R
  SPLIT_OP_RES_END = 5,        // R(dt/2) at P(t+3dt/4)
};

// Per-member constants of the local split-step operations.
template <typename T>
struct SplitConst {
  T inv_hbar, g_C, g_R, R, gamma_C, gamma_R;
  T noise_a, noise_b;
  unsigned long long seed;
  // Inactive-reservoir coupling, cross-spin term, two-field reservoir rates and the pump
  // share of each component (the cross-spin term and the shares are read by the IFRK
  // passes only).
  T g_I, alpha_2, gamma_I, gamma_A, R_IA, R_AI;
  T weight[2];
  T kappa;
};

struct RowPassArgs {
  int nx, ny, log2nx;
  int rows, log2rows;   // rows per block (power of two)
  int threads;
  int forward, inverse, multiply;
  int table_stride;     // complex values between consecutive members' propagator factors
  double scale;         // power-of-two factor of the kick: psi (1 + d) * scale
  const int* halt;      // steady-state monitor's halt word: when set the pass returns at once
};

struct ColPassArgs {
  int nx, ny, log2ny;
  int cols, log2cols;   // columns per block (power of two)
  int threads;
  int members;
  int forward, inverse;
  int op;               // SplitOp
  int reservoir;        // single reservoir present
  int res_kind;         // PG_RES_*: 2 double, 3 quadratic-double use the second field
  int potential;        // 0 none, 1 real, 2 complex
  int noise;
  long long pump_stride, pot_stride;
  int pump_terms;       // separable pump terms L
  long long pump_term_stride;  // reals between consecutive terms' envelopes
  int scale_offset;     // coefficient sample ([k][sample][term][member]) of the first coefficient
  int step_offset;      // noise step = step_base[0] + step_offset
  double dt_d;
  float dt_f;
  const int* halt;      // as RowPassArgs::halt
  // dt in the working precision is read through dt_of<T>().
  template <typename T>
  __host__ __device__ T dt_of() const;
};

template <>
inline __host__ __device__ float ColPassArgs::dt_of<float>() const { return dt_f; }
template <>
inline __host__ __device__ double ColPassArgs::dt_of<double>() const { return dt_d; }

template <typename T>
cudaError_t launch_row_pass(T* data, const T* tw, const T* px, const T* py, const RowPassArgs& a,
                            int members, cudaStream_t stream);

template <typename T>
cudaError_t launch_col_pass(T* data, T* res, const T* pump, const T* potential, const T* tw,
                            const SplitConst<T>* consts, const T* scales,
                            const unsigned long long* step_base, const ColPassArgs& a,
                            cudaStream_t stream);

template <typename T>
cudaError_t configure_split_kernels(size_t max_smem);

// The FP32 passes on register-resident transforms (split_reg.cu): axes of 64 to 4096 points.
inline bool reg_fft_size(int n) { return n >= 64 && n <= 4096 && (n & (n - 1)) == 0; }
// Values a thread holds of a transform of n points.  By size alone, so that a member's result does
// not depend on how many are stepped with it.  Eight to 512 points: a K-outer step of one 256^2 /
// 512^2 member 11.6 / 16.2 us against 17.9 / 21.5 with sixteen, eight 512^2 members 49.6 against
// 50.7 (sixteen is ahead only on large batches of small grids: 25.8 against 28.0 us for sixteen
// 256^2 members).  Above, two passes of eight do not reach n with a last DFT of at most 8.
inline int reg_fft_vals(int n) { return n <= 512 ? 8 : 16; }
// Attribute set-up for a grid's axes that have such passes, and launches.  tab: W_n^{t k} at entry
// k (n / vals) + t, k < vals, as {re, im} rounded and remainders.
cudaError_t configure_split_reg(int nx, int ny);
cudaError_t launch_row_reg(float* data, const float* tab, const float* px, const float* py,
                           const RowPassArgs& a, int members, int sm_count,
                           cudaStream_t stream);
cudaError_t launch_col_reg(float* data, float* res, const float* pump, const float* potential,
                           const float* tab, const SplitConst<float>* consts, const float* scales,
                           const unsigned long long* step_base, const ColPassArgs& a, int sm_count, cudaStream_t stream);

// The IFRK column pass for FP32 columns of 1024 sites on 32-value transforms (ifrk_col_fast.cu;
// one component, one single reservoir, one laser): whether a grid has it and whether it takes a
// launch, its W_1024^{n2 k1} table (1024 float4: rounded value, remainder), attribute set-up and
// launch.
struct IfrkRowArgs;
struct IfrkColArgs;
bool ifrk_col_fast_size(int nx, int ny);
bool ifrk_fast_col(const IfrkColArgs& a);
void ifrk_col_fast_twiddles(float* out);
cudaError_t configure_ifrk_col_fast();
cudaError_t launch_ifrk_col_fast(float* psi, const float* n0, float* dn_out, float* n_out,
                                 const float* psi_start, const float* psi_new, const float* pump,
                                 const float* potential, const float* tw4,
                                 const SplitConst<float>* consts, const float* scales,
                                 const unsigned long long* step_base, const IfrkColArgs& a,
                                 cudaStream_t stream);

// Complex values one thread stages per FFT pass: blocks need N * C <= this * threads.
int split_max_vals(bool is_double);

}  // namespace pg
