// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, FP32-flux EC volume flux, Rusanov surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec32_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC32, false, F_RUSANOV, false>(nq);
}
}  // namespace atb
