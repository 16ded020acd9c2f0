// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, FP32-flux EC volume flux, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec32_any(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC32, false, -1, false>(nq);
}
}  // namespace atb
