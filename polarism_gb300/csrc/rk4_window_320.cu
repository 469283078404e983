// The RK4 window kernel for windows of at most 320 columns.
#include "rk4_window.cuh"

namespace pg {

template decltype(launch_window_t<320>) launch_window_t<320>;

}  // namespace pg
