// fd_kernel instantiations (parallel compilation):
//   3-D Euler-gravity, FP32-flux Kennedy-Gruber volume flux, Rusanov surface flux
//   3-D Euler-gravity, FP32-flux Kennedy-Gruber volume flux, every surface flux
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_kg32_rus(int nq) {
  return fd_pick<LAW_EG, 3, VK_KG32, false, F_RUSANOV, false>(nq);
}
tend_launch_fn fd_eg3_kg32_any(int nq) {
  return fd_pick<LAW_EG, 3, VK_KG32, false, -1, false>(nq);
}
}  // namespace atb
