// fd_kernel instantiations (parallel compilation):
//   2-D Euler, EC volume flux, Rusanov surface flux
//   2-D Euler, FP32-flux EC volume flux, Rusanov surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_euler2_ec_rus(int nq) {
  return fd_pick<LAW_EULER, 2, VK_EC, false, F_RUSANOV, false>(nq);
}
tend_launch_fn fd_euler2_ec32_rus(int nq) {
  return fd_pick<LAW_EULER, 2, VK_EC32, false, F_RUSANOV, false>(nq);
}
}  // namespace atb
