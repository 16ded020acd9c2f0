// Which flux-differencing kernel serves an operator (atb_fd.cuh); nullptr when none is
// compiled for (law, dim, volume flux).  The kernels with the Rusanov flux as a
// compile-time constant carry no other numerical flux: fewer registers and a
// smaller instruction stream for the configurations that are run most.
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec_rus(int nq);
tend_launch_fn fd_eg3_ec_any(int nq);
tend_launch_fn fd_eg3_ec32_rus(int nq);
tend_launch_fn fd_eg3_ec32_any(int nq);
tend_launch_fn fd_eg3_kg_rus(int nq);
tend_launch_fn fd_eg3_kg_any(int nq);
tend_launch_fn fd_eg3_kg32_rus(int nq);
tend_launch_fn fd_eg3_kg32_any(int nq);
tend_launch_fn fd_eg3_weak_rus(int nq);
tend_launch_fn fd_eg3_weak_any(int nq);
tend_launch_fn fd_eg3_ec_fused_rus(int nq);
tend_launch_fn fd_eg3_ec_fused_any(int nq);
tend_launch_fn fd_eg3_ec32_fused_rus(int nq);
tend_launch_fn fd_eg3_ec32_fused_any(int nq);
tend_launch_fn fd_euler3_ec_any(int nq);
tend_launch_fn fd_euler2_ec_rus(int nq);
tend_launch_fn fd_euler2_ec32_rus(int nq);
tend_launch_fn fd_euler2_ec_any(int nq);
tend_launch_fn fd_euler2_ec32_any(int nq);
tend_launch_fn fd_eg2_ec_rus(int nq);
tend_launch_fn fd_eg2_ec_any(int nq);
tend_launch_fn fd_eg2_ec32_rus(int nq);
tend_launch_fn fd_eg2_ec32_any(int nq);
tend_launch_fn fd_sw2_ec_rus(int nq);
tend_launch_fn fd_sw2_ec32_rus(int nq);
tend_launch_fn fd_sw2_ec_any(int nq);
tend_launch_fn fd_sw2_ec32_any(int nq);
tend_launch_fn fd_eg3_ec_persist_rus(int nq);
tend_launch_fn fd_eg3_ec_fused_persist_rus(int nq);
tend_launch_fn fd_euler2_ec_persist_rus(int nq);
tend_launch_fn fd_sw2_ec_persist_rus(int nq);
tend_launch_fn fd_sw2_ec32_persist_rus(int nq);

tend_launch_fn pick_fd(int law, int dim, int vk, int nq, int sflux) {
  const bool rus = sflux == F_RUSANOV;
  if (law == LAW_EG && dim == 3) {
    if (vk == VK_EC) return rus ? fd_eg3_ec_rus(nq) : fd_eg3_ec_any(nq);
    if (vk == VK_EC32) return rus ? fd_eg3_ec32_rus(nq) : fd_eg3_ec32_any(nq);
    if (vk == VK_KG) return rus ? fd_eg3_kg_rus(nq) : fd_eg3_kg_any(nq);
    if (vk == VK_KG32) return rus ? fd_eg3_kg32_rus(nq) : fd_eg3_kg32_any(nq);
    if (vk == VK_WEAK) return rus ? fd_eg3_weak_rus(nq) : fd_eg3_weak_any(nq);
  }
  if (law == LAW_EG && dim == 2) {
    if (vk == VK_EC) return rus ? fd_eg2_ec_rus(nq) : fd_eg2_ec_any(nq);
    if (vk == VK_EC32) return rus ? fd_eg2_ec32_rus(nq) : fd_eg2_ec32_any(nq);
  }
  if (law == LAW_EULER && dim == 3 && vk == VK_EC) return fd_euler3_ec_any(nq);
  if (law == LAW_EULER && dim == 2) {
    if (vk == VK_EC) return rus ? fd_euler2_ec_rus(nq) : fd_euler2_ec_any(nq);
    if (vk == VK_EC32) return rus ? fd_euler2_ec32_rus(nq) : fd_euler2_ec32_any(nq);
  }
  if (law == LAW_SW && dim == 2) {
    if (vk == VK_EC) return rus ? fd_sw2_ec_rus(nq) : fd_sw2_ec_any(nq);
    if (vk == VK_EC32) return rus ? fd_sw2_ec32_rus(nq) : fd_sw2_ec32_any(nq);
  }
  return nullptr;
}

tend_launch_fn pick_fd_fused(int dim, int vk, int nq, int sflux, int lin_sflux) {
  if (dim != 3) return nullptr;
  const bool rus = sflux == F_RUSANOV && lin_sflux == F_RUSANOV;
  if (vk == VK_EC) return rus ? fd_eg3_ec_fused_rus(nq) : fd_eg3_ec_fused_any(nq);
  if (vk == VK_EC32) return rus ? fd_eg3_ec32_fused_rus(nq) : fd_eg3_ec32_fused_any(nq);
  return nullptr;
}

// persistent variants (atb_op_set_persistent): N = 3..5
tend_launch_fn pick_fd_persistent(int law, int dim, int vk, int nq, int sflux, bool fused, int lin_sflux) {
  if (nq < 4 || nq > 6 || sflux != F_RUSANOV || (fused && lin_sflux != F_RUSANOV)) return nullptr;
  if (fused) return (law == LAW_EG && dim == 3 && vk == VK_EC) ? fd_eg3_ec_fused_persist_rus(nq) : nullptr;
  if (law == LAW_EG && dim == 3 && vk == VK_EC) return fd_eg3_ec_persist_rus(nq);
  if (law == LAW_EULER && dim == 2 && vk == VK_EC) return fd_euler2_ec_persist_rus(nq);
  if (law == LAW_SW && dim == 2 && vk == VK_EC) return fd_sw2_ec_persist_rus(nq);
  if (law == LAW_SW && dim == 2 && vk == VK_EC32) return fd_sw2_ec32_persist_rus(nq);
  return nullptr;
}
}  // namespace atb
