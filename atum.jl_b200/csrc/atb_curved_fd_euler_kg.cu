// curved_fd_kernel instantiations (parallel compilation): Euler, Kennedy-Gruber volume flux, Rusanov or any surface flux
#include "atb_curved_fd.cuh"

namespace atb {
tend_launch_fn curved_fd_euler_kg_rus(int nq) { return curved_fd_pick<LAW_EULER, VK_KG, false, F_RUSANOV>(nq); }
tend_launch_fn curved_fd_euler_kg_any(int nq) { return curved_fd_pick<LAW_EULER, VK_KG, false, -1>(nq); }
}  // namespace atb
