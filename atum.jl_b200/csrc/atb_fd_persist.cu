// fd_kernel instantiations (parallel compilation):
//   2-D Euler, EC volume flux, persistent launches, Rusanov surface flux
//   2-D shallow water, EC volume flux, persistent launches, Rusanov surface flux
//   2-D shallow water, FP32-flux EC volume flux, persistent launches, Rusanov surface flux
//   3-D Euler-gravity, EC volume flux, fused ARK23 stage, persistent launches, Rusanov surface flux
//   3-D Euler-gravity, EC volume flux, persistent launches, Rusanov surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec_persist_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC, false, F_RUSANOV, true>(nq);
}
tend_launch_fn fd_eg3_ec_fused_persist_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_EC, true, F_RUSANOV, true>(nq);
}
tend_launch_fn fd_euler2_ec_persist_rus(int nq) {
  return fd_pick<LAW_EULER, 2, VK_EC, false, F_RUSANOV, true>(nq);
}
tend_launch_fn fd_sw2_ec_persist_rus(int nq) {
  return fd_pick<LAW_SW, 2, VK_EC, false, F_RUSANOV, true>(nq);
}
tend_launch_fn fd_sw2_ec32_persist_rus(int nq) {
  return fd_pick<LAW_SW, 2, VK_EC32, false, F_RUSANOV, true>(nq);
}
}  // namespace atb
