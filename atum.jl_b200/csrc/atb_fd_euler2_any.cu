// fd_kernel instantiations (parallel compilation):
//   2-D Euler, EC volume flux, every surface flux
//   2-D Euler, FP32-flux EC volume flux, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_euler2_ec_any(int nq) {
  return fd_pick<LAW_EULER, 2, VK_EC, false, -1, false>(nq);
}
tend_launch_fn fd_euler2_ec32_any(int nq) {
  return fd_pick<LAW_EULER, 2, VK_EC32, false, -1, false>(nq);
}
}  // namespace atb
