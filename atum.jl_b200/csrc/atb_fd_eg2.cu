// fd_kernel instantiations (parallel compilation):
//   2-D Euler-gravity, EC volume flux, Rusanov surface flux
//   2-D Euler-gravity, FP32-flux EC volume flux, Rusanov surface flux
//   2-D Euler-gravity, EC volume flux, every surface flux
//   2-D Euler-gravity, FP32-flux EC volume flux, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg2_ec_rus(int nq) {
  return fd_pick<LAW_EG, 2, VK_EC, false, F_RUSANOV, false>(nq);
}
tend_launch_fn fd_eg2_ec32_rus(int nq) {
  return fd_pick<LAW_EG, 2, VK_EC32, false, F_RUSANOV, false>(nq);
}
tend_launch_fn fd_eg2_ec_any(int nq) {
  return fd_pick<LAW_EG, 2, VK_EC, false, -1, false>(nq);
}
tend_launch_fn fd_eg2_ec32_any(int nq) {
  return fd_pick<LAW_EG, 2, VK_EC32, false, -1, false>(nq);
}
}  // namespace atb
