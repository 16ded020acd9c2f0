// Compile-time node-count specialisations of the tendency kernel: the weak form of
// linear Euler-gravity (the runtime-Nq kernel covers everything else).
#include "atb_tendency.cuh"
namespace atb {
static tend_launch_fn pick_nq_leg_3_vk_weak(int nq) {
  switch (nq) {
    case 3: return tend_launch<LAW_LEG, 3, VK_WEAK, 3>;
    case 4: return tend_launch<LAW_LEG, 3, VK_WEAK, 4>;
    case 5: return tend_launch<LAW_LEG, 3, VK_WEAK, 5>;
    case 6: return tend_launch<LAW_LEG, 3, VK_WEAK, 6>;
    case 7: return tend_launch<LAW_LEG, 3, VK_WEAK, 7>;
    case 8: return tend_launch<LAW_LEG, 3, VK_WEAK, 8>;
  }
  return nullptr;
}
static tend_launch_fn pick_nq_leg_2_vk_weak(int nq) {
  switch (nq) {
    case 3: return tend_launch<LAW_LEG, 2, VK_WEAK, 3>;
    case 4: return tend_launch<LAW_LEG, 2, VK_WEAK, 4>;
    case 5: return tend_launch<LAW_LEG, 2, VK_WEAK, 5>;
    case 6: return tend_launch<LAW_LEG, 2, VK_WEAK, 6>;
    case 7: return tend_launch<LAW_LEG, 2, VK_WEAK, 7>;
    case 8: return tend_launch<LAW_LEG, 2, VK_WEAK, 8>;
  }
  return nullptr;
}
tend_launch_fn pick_launcher_leg_nq(int dim, int vk, int nq) {
  if (vk != VK_WEAK) return nullptr;
  return dim == 3 ? pick_nq_leg_3_vk_weak(nq) : dim == 2 ? pick_nq_leg_2_vk_weak(nq) : nullptr;
}
}  // namespace atb
