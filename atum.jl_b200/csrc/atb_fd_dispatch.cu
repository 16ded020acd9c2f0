// Which flux-differencing kernel serves an operator (atb_fd.cuh); nullptr when none is
// compiled for (law, dim, volume flux).  The kernels with the Rusanov flux as a
// compile-time constant carry no other numerical flux: fewer registers and a
// smaller instruction stream for the configurations that are run most.
#include "atb_fd.cuh"

namespace atb {
tend_launch_fn fd_eg3_ec_rus(int nq);
tend_launch_fn fd_eg3_ec_any(int nq);
tend_launch_fn fd_eg3_kg_rus(int nq);
tend_launch_fn fd_eg3_kg_any(int nq);
tend_launch_fn fd_eg3_weak_rus(int nq);
tend_launch_fn fd_eg3_weak_any(int nq);
tend_launch_fn fd_eg3_ec_fused_rus(int nq);
tend_launch_fn fd_eg3_ec_fused_any(int nq);
tend_launch_fn fd_euler3_ec_any(int nq);
tend_launch_fn fd_euler2_ec_rus(int nq);
tend_launch_fn fd_euler2_ec_any(int nq);
tend_launch_fn fd_eg2_ec_rus(int nq);
tend_launch_fn fd_eg2_ec_any(int nq);
tend_launch_fn fd_sw2_ec_rus(int nq);
tend_launch_fn fd_sw2_ec32_rus(int nq);
tend_launch_fn fd_sw2_ec_any(int nq);
tend_launch_fn fd_sw2_ec32_any(int nq);
tend_launch_fn fd_eg3_ec_persist_rus(int nq);
tend_launch_fn fd_eg3_ec_fused_persist_rus(int nq);
tend_launch_fn fd_euler2_ec_persist_rus(int nq);
tend_launch_fn fd_sw2_ec_persist_rus(int nq);
tend_launch_fn fd_sw2_ec32_persist_rus(int nq);

// The FP32-flux forms of Euler and Euler-gravity run the FP64 pairs: an FP32 pair
// is 9 to 15 conversions from or to FP64, at a quarter of the rate of FP64
// arithmetic.  Measured on B200 per LSRK54 stage (Rusanov), FP32 pairs against
// FP64 pairs: 2-D Euler 8x8 elements N = 7, 17.5 and 6.9 us, 64x64 24.7 and
// 15.2; 3-D Euler-gravity EC 10^3 N = 4, 19.6 and 11.7; Kennedy-Gruber 26.9 and
// 9.2: FP64 was the faster one at every order N = 1..7 and size, by 1.3 to 2.9.
// Shallow water, within 20 % of FP64, keeps its own.
int fd_volume_kind(int law, int vk) {
  if (law == LAW_SW) return vk;
  return vk == VK_EC32 ? VK_EC : vk == VK_KG32 ? VK_KG : vk;
}

tend_launch_fn pick_fd(int law, int dim, int vk, int nq, int sflux) {
  vk = fd_volume_kind(law, vk);
  const bool rus = sflux == F_RUSANOV;
  if (law == LAW_EG && dim == 3) {
    if (vk == VK_EC) return rus ? fd_eg3_ec_rus(nq) : fd_eg3_ec_any(nq);
    if (vk == VK_KG) return rus ? fd_eg3_kg_rus(nq) : fd_eg3_kg_any(nq);
    if (vk == VK_WEAK) return rus ? fd_eg3_weak_rus(nq) : fd_eg3_weak_any(nq);
  }
  if (law == LAW_EG && dim == 2 && vk == VK_EC) return rus ? fd_eg2_ec_rus(nq) : fd_eg2_ec_any(nq);
  if (law == LAW_EULER && dim == 3 && vk == VK_EC) return fd_euler3_ec_any(nq);
  if (law == LAW_EULER && dim == 2 && vk == VK_EC) return rus ? fd_euler2_ec_rus(nq) : fd_euler2_ec_any(nq);
  if (law == LAW_SW && dim == 2) {
    if (vk == VK_EC) return rus ? fd_sw2_ec_rus(nq) : fd_sw2_ec_any(nq);
    if (vk == VK_EC32) return rus ? fd_sw2_ec32_rus(nq) : fd_sw2_ec32_any(nq);
  }
  return nullptr;
}

tend_launch_fn pick_fd_fused(int dim, int vk, int nq, int sflux, int lin_sflux) {
  if (dim != 3 || (vk != VK_EC && vk != VK_EC32)) return nullptr;
  const bool rus = sflux == F_RUSANOV && lin_sflux == F_RUSANOV;
  return rus ? fd_eg3_ec_fused_rus(nq) : fd_eg3_ec_fused_any(nq);
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
