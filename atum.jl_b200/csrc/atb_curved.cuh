// Curved-element (cubed-sphere) DGSEM tendency kernels: host-side entry points.
#pragma once
#include "atb_tendency.cuh"

namespace atb {

// Node-per-thread kernels (atb_curved.cu): dynamic shared memory of E elements;
// it also bounds the elements per CTA that an operator accepts
size_t curved_smem_bytes(int vk, int naux, int Nq, int E);
// Launcher for (law, volume kind, surface flux) at any order; nullptr when
// there is none (Euler, Euler-gravity, linear Euler-gravity: weak, central)
tend_launch_fn pick_launcher_curved(int law, int vk, int sflux);

// Line-per-thread kernels (atb_curved_fd.cuh): Euler and Euler-gravity, EC and
// KG volume fluxes, 2 <= Nq <= 8
int curved_fd_elements(int Nq);  // most elements per CTA
size_t curved_fd_smem_bytes(int Nq, int E, bool fuse);
tend_launch_fn pick_curved_fd(int law, int vk, int Nq, int sflux);
// the fused ARK23 stage (Euler-gravity EC / KG + radial weak-form linear
// Euler-gravity, Rusanov faces of both); nullptr when there is none
tend_launch_fn pick_curved_fd_fused(int vk, int Nq, int sflux, int lin_sflux);

}  // namespace atb
