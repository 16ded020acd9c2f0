// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, EC volume flux, fused ARK23 stage, Rusanov surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec_fused_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC, true, F_RUSANOV, false>(nq);
}
}  // namespace atb
