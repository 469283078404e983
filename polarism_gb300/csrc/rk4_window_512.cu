// The RK4 window kernel for windows of at most 512 columns.
#include "rk4_window.cuh"

namespace pg {

template decltype(launch_window_t<512>) launch_window_t<512>;

}  // namespace pg
