// fd_kernel instantiations (parallel compilation):
//   3-D Euler, EC volume flux, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_euler3_ec_any(int nq) {
  return fd_pick<LAW_EULER, 3, VK_EC, false, -1, false>(nq);
}
}  // namespace atb
