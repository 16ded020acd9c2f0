// Dispatch to the compile-time node-count specialisations (atb_knq_*.cu).
#include "atb_tendency.cuh"
namespace atb {
tend_launch_fn pick_nq_leg_3_vk_weak(int nq);
tend_launch_fn pick_nq_leg_2_vk_weak(int nq);
template <> tend_launch_fn pick_launcher_nq<LAW_ADV>(int dim, int vk, int nq) {
  (void)dim; (void)vk; (void)nq;
  return nullptr;
}
template <> tend_launch_fn pick_launcher_nq<LAW_EULER>(int dim, int vk, int nq) {
  (void)dim; (void)vk; (void)nq;
  return nullptr;
}
template <> tend_launch_fn pick_launcher_nq<LAW_EG>(int dim, int vk, int nq) {
  (void)dim; (void)vk; (void)nq;
  return nullptr;
}
template <> tend_launch_fn pick_launcher_nq<LAW_LEG>(int dim, int vk, int nq) {
  if (dim == 3 && vk == VK_WEAK) return pick_nq_leg_3_vk_weak(nq);
  if (dim == 2 && vk == VK_WEAK) return pick_nq_leg_2_vk_weak(nq);
  (void)dim; (void)vk; (void)nq;
  return nullptr;
}
template <> tend_launch_fn pick_launcher_nq<LAW_SW>(int dim, int vk, int nq) {
  (void)dim; (void)vk; (void)nq;
  return nullptr;
}
}  // namespace atb
