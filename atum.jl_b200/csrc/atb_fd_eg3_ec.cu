// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, EC volume flux, Rusanov surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC, false, F_RUSANOV, false>(nq);
}
}  // namespace atb
