// The RK4 window kernel for windows of at most 1024 columns.
#include "rk4_window.cuh"

namespace pg {

template decltype(launch_window_t<1024>) launch_window_t<1024>;

}  // namespace pg
