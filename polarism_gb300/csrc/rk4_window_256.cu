// The RK4 window kernel for windows of at most 256 columns.
#include "rk4_window.cuh"

namespace pg {

template decltype(launch_window_t<256>) launch_window_t<256>;

}  // namespace pg
