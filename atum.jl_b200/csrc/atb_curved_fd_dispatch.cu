// Which line-per-thread kernel serves an operator on curved elements
// (atb_curved_fd.cuh), and its launch sizes.
#include "atb_curved_fd.cuh"

namespace atb {
tend_launch_fn curved_fd_eg_ec_rus(int nq);
tend_launch_fn curved_fd_eg_ec_any(int nq);
tend_launch_fn curved_fd_eg_kg_rus(int nq);
tend_launch_fn curved_fd_eg_kg_any(int nq);
tend_launch_fn curved_fd_euler_ec_rus(int nq);
tend_launch_fn curved_fd_euler_ec_any(int nq);
tend_launch_fn curved_fd_euler_kg_rus(int nq);
tend_launch_fn curved_fd_euler_kg_any(int nq);
tend_launch_fn curved_fd_eg_ec_fused(int nq);
tend_launch_fn curved_fd_eg_kg_fused(int nq);

int curved_fd_elements(int nq) {
  const int m = curved_fd_cfg(nq).max_threads / line_count(nq, 3);
  return m < 1 ? 1 : m;
}

size_t curved_fd_smem_bytes(int nq, int E, bool fuse) {
  return sizeof(double) * (size_t)E * curved_fd_slot(nq, fuse);
}

tend_launch_fn pick_curved_fd(int law, int vk, int nq, int sflux) {
  const bool rus = sflux == F_RUSANOV;
  if (law == LAW_EG) {
    if (vk == VK_EC) return rus ? curved_fd_eg_ec_rus(nq) : curved_fd_eg_ec_any(nq);
    if (vk == VK_KG) return rus ? curved_fd_eg_kg_rus(nq) : curved_fd_eg_kg_any(nq);
  } else if (law == LAW_EULER) {
    if (vk == VK_EC) return rus ? curved_fd_euler_ec_rus(nq) : curved_fd_euler_ec_any(nq);
    if (vk == VK_KG) return rus ? curved_fd_euler_kg_rus(nq) : curved_fd_euler_kg_any(nq);
  }
  return nullptr;
}

tend_launch_fn pick_curved_fd_fused(int vk, int nq, int sflux, int lin_sflux) {
  if (sflux != F_RUSANOV || lin_sflux != F_RUSANOV) return nullptr;
  return vk == VK_EC ? curved_fd_eg_ec_fused(nq) : vk == VK_KG ? curved_fd_eg_kg_fused(nq) : nullptr;
}
}  // namespace atb
