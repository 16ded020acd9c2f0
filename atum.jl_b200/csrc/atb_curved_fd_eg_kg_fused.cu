// curved_fd_kernel instantiations (parallel compilation): fused ARK23 stage, Euler-gravity, Kennedy-Gruber volume flux
#include "atb_curved_fd.cuh"

namespace atb {
tend_launch_fn curved_fd_eg_kg_fused(int nq) { return curved_fd_pick<LAW_EG, VK_KG, true, F_RUSANOV>(nq); }
}  // namespace atb
