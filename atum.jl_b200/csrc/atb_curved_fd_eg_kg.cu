// curved_fd_kernel instantiations (parallel compilation): Euler-gravity, Kennedy-Gruber volume flux, Rusanov or any surface flux
#include "atb_curved_fd.cuh"

namespace atb {
tend_launch_fn curved_fd_eg_kg_rus(int nq) { return curved_fd_pick<LAW_EG, VK_KG, false, F_RUSANOV>(nq); }
tend_launch_fn curved_fd_eg_kg_any(int nq) { return curved_fd_pick<LAW_EG, VK_KG, false, -1>(nq); }
}  // namespace atb
