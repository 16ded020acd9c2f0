// DGSEM tendency on curved hexahedra (cubed-sphere shells): per-node metric
// terms, per-face-node normals and face masses, neighbour traces through a
// node-level face map.
//
// Restates, for one stage, src/dgsem.jl:217-306 (volumeterm!, weak form),
// 470-561 (esvolumeterm_dir!, flux differencing: l_g = MJ g[dir, :] of both
// nodes of every pair, all three rows of the two-point flux contracted with
// them) and 683-732 (surfaceterm! with facenormal / faceMJ / faceix of a curved
// grid), with the same epilogues as the brick kernels (atb_tendency.cuh).
//
// Mapping: one thread per LGL node, E elements per CTA.  The element's state
// and aux, the per-node values the volume term reads of other nodes (weak
// form: the contravariant flux rows MJ g[dir, :] . F; central flux
// differencing: MJ g) are staged in shared memory.  Face tasks evaluate the numerical flux once per face node,
// gather the neighbour trace from global memory and leave faceMJ * flux in a
// shared slot; every node then subtracts the slots of its faces in face order.
// The entropy-conservative and Kennedy-Gruber volume fluxes run one thread per
// line (atb_curved_fd.cuh); brick grids have their own kernels (diagonal
// metrics, one flux row).
#include "atb_curved_flux.cuh"

namespace atb {

namespace {

// per-node values staged for other nodes of the element: central flux
// differencing stages MJ g (9); the weak form the contravariant flux rows (3 x NS)
template <int VK> struct CurvedX {
  static constexpr int v = (VK == VK_WEAK) ? 3 * CNS : 9;
};

// SF >= 0: the surface flux kind as a compile-time constant (the kernel then
// carries no other flux's code); SF < 0: the kind given at run time.
template <int LAW, int VK, int SF>
__global__ void __launch_bounds__(512) curved_kernel(const TendArgs A) {
  constexpr int NS = CNS;
  constexpr int NA = NAuxMax<LAW, 3>::v;
  constexpr int NX = CurvedX<VK>::v;
  extern __shared__ __align__(16) double smem[];
  const int Nq = A.Nq, Np = A.Np, Nfp = A.Nfp, E = A.E, na = A.naux;
  const int nqq = (Nq * Nq + 1) & ~1;
  double* sD = smem;  // D[i][m] = l_m'(xi_i)
  const size_t per = (size_t)(NS + na + NX) * Np + (size_t)6 * Nfp * NS;
  const int tid = threadIdx.x;
  const int el = tid / Np;
  const int node = tid - el * Np;
  const int e = blockIdx.x * E + el;
  const bool active = el < E && e < A.K;
  for (int i = tid; i < Nq * Nq; i += blockDim.x) sD[i] = A.Dmat[i];
  // the state, aux and accumulators below may come from the previous kernel
  // of the stream (programmatic dependent launch, launch_maybe_pdl)
  pdl_wait();
  double* base = smem + nqq + (size_t)(el < E ? el : 0) * per;
  double* sq = base;
  double* sa = sq + (size_t)NS * Np;
  double* sx = sa + (size_t)na * Np;
  const size_t stride = A.stride;
  const size_t gid = (size_t)e * Np + node;
  double qn[NS], an[NA];
#pragma unroll
  for (int k = 0; k < NA; ++k) an[k] = 0.0;
  double MJ = 1.0, lg[3][3];
  if (active) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      qn[s] = A.q[s][gid];
      sq[s * Np + node] = qn[s];
    }
    for (int k = 0; k < na && k < NA; ++k) {
      an[k] = A.aux[(size_t)k * stride + gid];
      sa[k * Np + node] = an[k];
    }
    MJ = A.MJn[gid];
    // metric terms of the active directions only (the radial linear operator
    // of the IMEX stages reads a third of them)
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int c = 0; c < 3; ++c) lg[d][c] = ((A.dirs >> d) & 1) ? A.G[((size_t)d * 3 + c) * stride + gid] : 0.0;
    if constexpr (VK == VK_WEAK) {
      double F[3][NS];
      flux_rows<LAW>(A.law, qn, an, F);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (!((A.dirs >> d) & 1)) continue;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          double acc = 0.0;
#pragma unroll
          for (int c = 0; c < 3; ++c) acc = acc + lg[d][c] * F[c][s];
          sx[(d * NS + s) * Np + node] = acc * MJ;
        }
      }
    } else {
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          lg[d][c] = MJ * lg[d][c];
          sx[(d * 3 + c) * Np + node] = lg[d][c];
        }
    }
  }
  __syncthreads();

  // ---------------------------------------------------------- face tasks
  const int ntask = E * 6 * Nfp;
  for (int t = tid; t < ntask; t += blockDim.x) {
    const int fe = t / (6 * Nfp);
    const int r = t - fe * 6 * Nfp;
    const int face = r / Nfp, j = r - face * Nfp;
    const int k = face >> 1, side = face & 1;
    const int eg = blockIdx.x * E + fe;
    if (eg >= A.K || !((A.dirs >> k) & 1)) continue;
    // face node j: tangential dimensions in increasing order, first fastest
    const int t0 = j % Nq, t1 = j / Nq;
    const int ek = side ? Nq - 1 : 0;
    const int fn = (k == 0) ? ek + Nq * (t0 + Nq * t1) : (k == 1) ? t0 + Nq * (ek + Nq * t1) : t0 + Nq * (t1 + Nq * ek);
    double* fb = smem + nqq + (size_t)fe * per;
    const double* fq = fb;
    const double* fa = fb + (size_t)NS * Np;
    double* slot = fb + (size_t)(NS + na + NX) * Np;
    const size_t fj = ((size_t)eg * 6 + face) * Nfp + j;
    double n[3], qm[NS], am[NA], qp[NS], ap[NA];
#pragma unroll
    for (int c = 0; c < 3; ++c) n[c] = A.fnrm[fj * 3 + c];
#pragma unroll
    for (int s = 0; s < NS; ++s) qm[s] = fq[s * Np + fn];
#pragma unroll
    for (int c = 0; c < NA; ++c) am[c] = ap[c] = 0.0;
    for (int c = 0; c < na && c < NA; ++c) am[c] = fa[c * Np + fn];
    const int nb = A.fnb[fj];
    if (nb >= 0) {
#pragma unroll
      for (int s = 0; s < NS; ++s) qp[s] = A.q[s][nb];
      for (int c = 0; c < na && c < NA; ++c) ap[c] = A.aux[(size_t)c * stride + nb];
    } else {
      boundary_state_n(A.law, n, -1 - nb, qm, qp);
#pragma unroll
      for (int c = 0; c < NA; ++c) ap[c] = am[c];
    }
    double nf[NS];
    surface_flux_n<LAW>(A.law, SF >= 0 ? SF : A.sflux, n, qm, am, qp, ap, nf);
    const double fm = A.fMJ[fj];
#pragma unroll
    for (int s = 0; s < NS; ++s) slot[(face * Nfp + j) * NS + s] = fm * nf[s];
  }
  __syncthreads();
  if (!active) return;

  // ------------------------------------------------------------- volume
  const double MJI = 1.0 / MJ;
  int ijk[3] = {node % Nq, (node / Nq) % Nq, node / (Nq * Nq)};
  double T[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) T[s] = -0.0;
  if ((A.dirs >> 2) & 1) add_sources<LAW, 3>(A.law, VK == VK_WEAK, qn, an, T);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!((A.dirs >> d) & 1)) continue;
    const int i = ijk[d];
    const int step = (d == 0) ? 1 : (d == 1) ? Nq : Nq * Nq;
    const int n0 = node - i * step;
    if constexpr (VK == VK_WEAK) {
      for (int m = 0; m < Nq; ++m) {
        const double Dm = sD[m * Nq + i] * MJI;
        const int nn = n0 + m * step;
#pragma unroll
        for (int s = 0; s < NS; ++s) T[s] = T[s] + Dm * sx[(d * NS + s) * Np + nn];
      }
    } else {
      for (int m = 0; m < Nq; ++m) {
        if (m == i) continue;  // -D_ii lg_i F + F lg_i D_ii: no contribution
        const int nn = n0 + m * step;
        double q2[NS], a2[NA], F[3][NS], f1[NS], f2[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) q2[s] = sq[s * Np + nn];
#pragma unroll
        for (int c = 0; c < NA; ++c) a2[c] = 0.0;
        for (int c = 0; c < na && c < NA; ++c) a2[c] = sa[c * Np + nn];
        twopoint_rows<LAW, VK>(A.law, qn, an, nullptr, q2, a2, nullptr, F);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          f1[s] = lg[d][0] * F[0][s] + lg[d][1] * F[1][s] + lg[d][2] * F[2][s];
          f2[s] = sx[d * 3 * Np + nn] * F[0][s] + sx[(d * 3 + 1) * Np + nn] * F[1][s] + sx[(d * 3 + 2) * Np + nn] * F[2][s];
        }
        const double Ddn = MJI * sD[i * Nq + m], Dnd = MJI * sD[m * Nq + i];
#pragma unroll
        for (int s = 0; s < NS; ++s) T[s] = T[s] - Ddn * f1[s] + Dnd * f2[s];
      }
    }
  }
  // ------------------------------------------------------------ surface
  const double* slot = sx + (size_t)NX * Np;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (!((A.dirs >> k) & 1)) continue;
    const int id = ijk[k];
    if (id != 0 && id != Nq - 1) continue;
    const int side = (id == Nq - 1) ? 1 : 0;
    const int j = (k == 0) ? ijk[1] + Nq * ijk[2] : (k == 1) ? ijk[0] + Nq * ijk[2] : ijk[0] + Nq * ijk[1];
    const int face = 2 * k + side;
#pragma unroll
    for (int s = 0; s < NS; ++s) T[s] = T[s] - slot[(face * Nfp + j) * NS + s] * MJI;
  }

  // ----------------------------------------------------------- epilogue
  switch (A.epi) {
    case EPI_SET:
#pragma unroll
      for (int s = 0; s < NS; ++s) A.out[s][gid] = T[s];
      break;
    case EPI_ADD:
#pragma unroll
      for (int s = 0; s < NS; ++s) A.out[s][gid] = A.out[s][gid] + T[s];
      break;
    case EPI_LSRK: {
      const double bdt = A.dte ? A.bdt * A.dte[e] : A.bdt;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double dqn = (A.a != 0.0) ? A.a * A.out[s][gid] + T[s] : T[s];
        A.out[s][gid] = dqn;
        A.out2[s][gid] = qn[s] + bdt * dqn;
      }
    } break;
    case EPI_ARK:
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        // out holds N(Q), T = L(Q)
        const double Ex = A.out[s][gid] - T[s];
#pragma unroll
        for (int jj = 0; jj < 3; ++jj)
          if (A.acc[jj][0]) {
            const double b0 = A.accin[jj][0] ? A.accin[jj][s][gid] : qn[s];
            A.acc[jj][s][gid] = b0 + A.adt * (A.ca[jj] * Ex + A.cb[jj] * T[s]);
          }
      }
      break;
    case EPI_SUBOUT2:
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double o2 = A.out2[s][gid];
        A.out[s][gid] = T[s];
        A.out2[s][gid] = o2 - T[s];
      }
      break;
    case EPI_RLSRK:
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double o2 = A.out2[s][gid];
        A.out[s][gid] = T[s];
        A.out2[s][gid] = A.a * o2 + T[s];
      }
      break;
  }
  pdl_trigger();
}

template <int LAW, int VK, int SF>
void curved_launch(const TendArgs& A, int grid, int block, size_t smem, cudaStream_t st) {
  static SmemLimit limit;
  raise_smem(curved_kernel<LAW, VK, SF>, limit, smem);
  launch_maybe_pdl(curved_kernel<LAW, VK, SF>, dim3(grid), dim3(block), smem, st, A);
}

}  // namespace

size_t curved_smem_bytes(int vk, int naux, int Nq, int E) {
  const int Np = Nq * Nq * Nq, Nfp = Nq * Nq;
  const int nx = (vk == VK_WEAK) ? 3 * CNS : NPreE<3>::v + 9;
  return sizeof(double) * ((size_t)((Nq * Nq + 1) & ~1) + ((size_t)(CNS + naux + nx) * Np + (size_t)6 * Nfp * CNS) * E);
}

tend_launch_fn pick_launcher_curved(int law, int vk, int sflux) {
  // Rusanov (the sphere experiments' surface flux) built in; every other
  // surface flux through the run-time kind
  const bool rus = sflux == F_RUSANOV;
  switch (law) {
    case LAW_EULER:
      if (vk == VK_WEAK) return rus ? curved_launch<LAW_EULER, VK_WEAK, F_RUSANOV> : curved_launch<LAW_EULER, VK_WEAK, -1>;
      if (vk == VK_CENTRAL) return curved_launch<LAW_EULER, VK_CENTRAL, -1>;
      break;
    case LAW_EG:
      if (vk == VK_WEAK) return rus ? curved_launch<LAW_EG, VK_WEAK, F_RUSANOV> : curved_launch<LAW_EG, VK_WEAK, -1>;
      if (vk == VK_CENTRAL) return curved_launch<LAW_EG, VK_CENTRAL, -1>;
      break;
    case LAW_LEG:
      if (vk == VK_WEAK) return rus ? curved_launch<LAW_LEG, VK_WEAK, F_RUSANOV> : curved_launch<LAW_LEG, VK_WEAK, -1>;
      if (vk == VK_CENTRAL) return curved_launch<LAW_LEG, VK_CENTRAL, -1>;
      break;
  }
  return nullptr;
}

}  // namespace atb
