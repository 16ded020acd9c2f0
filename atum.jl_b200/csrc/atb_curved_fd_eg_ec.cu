// curved_fd_kernel instantiations (parallel compilation): Euler-gravity, entropy-conservative volume flux, Rusanov or any surface flux
#include "atb_curved_fd.cuh"

namespace atb {
tend_launch_fn curved_fd_eg_ec_rus(int nq) { return curved_fd_pick<LAW_EG, VK_EC, false, F_RUSANOV>(nq); }
tend_launch_fn curved_fd_eg_ec_any(int nq) { return curved_fd_pick<LAW_EG, VK_EC, false, -1>(nq); }
}  // namespace atb
