// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, weak form, Rusanov surface flux
//   3-D Euler-gravity, weak form, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_weak_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_WEAK, false, F_RUSANOV, false>(nq);
}
tend_launch_fn fd_eg3_weak_any(int nq) {
  return fd_pick<LAW_EG, 3, VK_WEAK, false, -1, false>(nq);
}
}  // namespace atb
