// Flux-differencing tendency on curved hexahedra, one thread per tensor line
// (atb_fd.cuh's scheme on per-node metric terms; atb_curved.cu describes the
// operator and serves the weak and central forms).
//
// With l_a = M J g[d, :] at node a, the reference's contraction of the
// symmetric two-point flux F#(a, b) (src/dgsem.jl:497-553),
//   M J dT_a = sum_b  D_ba l_b . F# - D_ab l_a . F#  =  sum_b w . F#,
//   w = D_ba l_b - D_ab l_a,
// changes sign when a and b change places: one contraction serves both nodes
// (the Euler-gravity fluctuation, scaled by the node's own p/rho, keeps its
// sign).  The contraction is closed: U = w . u_avg, f_rho = U rho_log, momentum
// f_rho u_avg + p_c w, energy f_rho (...) + p_c U.  1/(M J) is applied once, to
// the finished sums.
//
// What bounds it: issue and latency at 12 warps per SM (registers); the FP64
// pipe is 38 % busy, the pairs take half of its work and the staging, faces and
// epilogue the rest.  Measured on B200 against the kernel with one thread per
// node and ordered pairs: 3000 shell elements at N = 5, fused ARK23 stage 262 ->
// 133 us; 750 at N = 3, LSRK54 stage 15.9 -> 9.1 us.
#pragma once
#include "atb_curved_flux.cuh"
#include "atb_fd.cuh"

namespace atb {

// Largest CTA and resident CTAs (atb_fd.cuh, FdCfg).  Measured at Nq = 6 (fused
// stage): 3 CTAs of 128 threads 133 us, 4 of 128 (128 registers, spills) 151,
// 2 of 224 142; without reading a line's values again per pair 143.  Nq = 4: 2
// of 224, 3 of 144, 3 of 160 and 5 of 96 within 1 %.
__host__ __device__ constexpr FdCfg curved_fd_cfg(int nq) {
  if (nq == 8) return FdCfg{192, 2, 1};
  if (nq == 7) return FdCfg{160, 2, 1};
  if (nq == 6) return FdCfg{128, 3, 1};
  if (nq == 5) return FdCfg{160, 3, 1};
  return FdCfg{224, 2, 1};
}
// point values: u/2 (3), B = rho/p (KG: p/2), Phi/4, p/rho (KG: e/2); then M J g (9)
constexpr int CFD_NP = 6, CFD_NX = CFD_NP + 9;
// doubles per element: state, point values (the three directions' sums reuse
// them); fused: linear p', H, the linear tendency's sums
__host__ __device__ constexpr int curved_fd_slot(int nq, bool fuse) {
  return (5 + CFD_NX + (fuse ? 2 + 5 : 0)) * line_nodes(nq, 3);
}
static_assert(CFD_NX >= 3 * 5, "the sums of three directions fit the point values' region");

struct CurvedPt {
  double r, v[3], w, ph, x, l[3];
};
template <int LAW, bool VOL>
__device__ __forceinline__ void curved_load(CurvedPt& P, const double* sq_, const double* sx_, int npl, int n, int d) {
  using Ptr = std::conditional_t<VOL, const volatile double*, const double*>;
  const Ptr sq = sq_, sx = sx_;
  P.r = sq[n];
#pragma unroll
  for (int c = 0; c < 3; ++c) P.v[c] = sx[c * npl + n];
  P.w = sx[3 * npl + n];
  if constexpr (LAW == LAW_EG) P.ph = sx[4 * npl + n];
  P.x = sx[5 * npl + n];
#pragma unroll
  for (int c = 0; c < 3; ++c) P.l[c] = sx[(CFD_NP + 3 * d + c) * npl + n];
}

// adds the pair's contraction to both nodes (dab = D[a][b], dba = D[b][a])
template <int LAW, int VK, int TIER>
__device__ __forceinline__ void curved_pair(double c0, double dab, double dba, const CurvedPt& P, const CurvedPt& Q,
                                            double* Ta, double* Tb) {
  double w[3], ua[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w[c] = fma(-dab, P.l[c], __dmul_rn(dba, Q.l[c]));
    ua[c] = P.v[c] + Q.v[c];
  }
  const double U = dot<3>(w, ua);
  double rl, pc, ef, fa = 0.0, fb = 0.0;
  if constexpr (VK == VK_KG) {
    rl = 0.5 * (P.r + Q.r);
    pc = P.w + Q.w;
    ef = P.x + Q.x;
    if constexpr (LAW == LAW_EG) {
      fa = __dmul_rn(rl, 2.0 * (P.ph - Q.ph));  // rho_avg / 2 (Phi_a - Phi_b)
      fb = -fa;
    }
  } else {
    const double R = P.r + Q.r, rd = P.r - Q.r, B = P.w + Q.w, bd = P.w - Q.w;
    double ct;
    if constexpr (TIER < 2) {
      const double R2 = R * R, B2 = B * B;
      const double inv = rcp_cheb(R2 * B2);
      const double ib2 = R2 * inv, ir2 = B2 * inv, iB = B * ib2;
      const double ur = (rd * rd) * ir2, ub = (bd * bd) * ib2;
      rl = TIER == 0 ? R * mean_Gh(ur) : (0.5 * R) * rcp_cheb(mean_F_wide(ur));
      ct = (TIER == 0 ? mean_F(ub) : mean_F_wide(ub)) * (iB * c0);
      pc = R * iB;
    } else {
      const double iB = 1.0 / B;
      rl = logavg_wide(P.r, Q.r);
      pc = R * iB;
      ct = 0.5 * c0 / logavg_wide(P.w, Q.w);
    }
    ef = fma(2.0, dot<3>(P.v, Q.v), ct);
    if constexpr (LAW == LAW_EG) {
      ef = fma(2.0, P.ph + Q.ph, ef);
      const double x = __dmul_rn(__dmul_rn(B, rl), P.ph - Q.ph);  // b_avg rho_log (Phi_a - Phi_b)
      fa = __dmul_rn(P.x, x);
      fb = -__dmul_rn(Q.x, x);
    }
  }
  const double fr = __dmul_rn(U, rl);
  Ta[0] += fr;
  Tb[0] -= fr;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double m = __dmul_rn(fr, ua[c]);
    if constexpr (LAW == LAW_EG) {
      Ta[1 + c] += fma(pc - fa, w[c], m);
      Tb[1 + c] -= fma(pc - fb, w[c], m);
    } else {
      const double f = fma(pc, w[c], m);
      Ta[1 + c] += f;
      Tb[1 + c] -= f;
    }
  }
  const double fe = fma(fr, ef, __dmul_rn(pc, U));
  Ta[4] += fe;
  Tb[4] -= fe;
}

template <int LAW, int VK, int NQ, int TIER>
__device__ __forceinline__ void curved_pairs(const TendArgs& A, double c0, const double* sq, const double* sx, int base,
                                             int sd, int d, double (*T)[5]) {
  constexpr int npl = line_nodes(NQ, 3);
#pragma unroll
  for (int a = 0; a < NQ - 1; ++a) {
    CurvedPt P;
    curved_load<LAW, (NQ >= 5)>(P, sq, sx, npl, base + a * sd, d);
#pragma unroll
    for (int b = a + 1; b < NQ; ++b) {
      CurvedPt Q;
      curved_load<LAW, (NQ >= 5)>(Q, sq, sx, npl, base + b * sd, d);
      curved_pair<LAW, VK, TIER>(c0, A.cfd[a * NQ + b], A.cfd[b * NQ + a], P, Q, T[a], T[b]);
    }
  }
}

// Rusanov flux . n (src/numericalfluxes.jl:31-42) for a unit normal, from one
// reciprocal of the density per side
template <int LAW>
__device__ __forceinline__ void curved_rusanov(const LawP& L, const double* n, const double* qm, double Pm,
                                               double dpm, const double* qp, double Pp, double dpp, double* nf) {
  const double rm = rcp_cheb(qm[0]), rp = rcp_cheb(qp[0]);
  const double mm = dot<3>(qm + 1, n), mp = dot<3>(qp + 1, n);
  const double um = __dmul_rn(mm, rm), up = __dmul_rn(mp, rp), g1 = L.gamma - 1.0;
  double tm = fma(__dmul_rn(-0.5, rm), dot<3>(qm + 1, qm + 1), qm[4]);
  double tp = fma(__dmul_rn(-0.5, rp), dot<3>(qp + 1, qp + 1), qp[4]);
  if constexpr (LAW == LAW_EG) {
    tm = fma(-qm[0], Pm, tm);
    tp = fma(-qp[0], Pp, tp);
  }
  const double pm = __dmul_rn(g1, tm), pp = __dmul_rn(g1, tp);
  const double cm = sqrt_house(__dmul_rn(__dmul_rn(L.gamma, pm), rm));
  const double cp = sqrt_house(__dmul_rn(__dmul_rn(L.gamma, pp), rp));
  const double ws = -0.5 * dmax(fabs(um) + cm, fabs(up) + cp);
  const double ps = (pm - dpm) + (pp - dpp);
  nf[0] = fma(ws, qp[0] - qm[0], 0.5 * (mm + mp));
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double f = fma(um, qm[1 + c], fma(up, qp[1 + c], __dmul_rn(ps, n[c])));
    nf[1 + c] = fma(ws, qp[1 + c] - qm[1 + c], 0.5 * f);
  }
  const double fe = fma(um, qm[4] + pm, __dmul_rn(up, qp[4] + pp));
  nf[4] = fma(ws, qp[4] - qm[4], 0.5 * fe);
}

// every surface flux, chosen at run time: one out-of-line copy
template <int LAW>
__device__ __noinline__ void curved_flux_any(const LawP& L, int kind, const double* n, const double* qm,
                                             const double* am, const double* qp, const double* ap, double* nf) {
  surface_flux_n<LAW>(L, kind, n, qm, am, qp, ap, nf);
}

template <int LAW, int VK, int NQ, bool FUSE, int SF>
__global__ void __launch_bounds__(curved_fd_cfg(NQ).max_threads, curved_fd_cfg(NQ).min_blocks)
    curved_fd_kernel(const __grid_constant__ TendArgs A) {
  constexpr int NS = 5, ROW = line_row(NQ), NPL = line_nodes(NQ, 3), NP = NQ * NQ * NQ, NFP = NQ * NQ;
  constexpr int slotsz = curved_fd_slot(NQ, FUSE);
  constexpr int OX = NS * NPL, OL = OX + CFD_NX * NPL, OT = OL + 2 * NPL;
  constexpr bool EG = LAW == LAW_EG;
  constexpr int NA = NAuxMax<LAW, 3>::v;
  constexpr int RN = (NQ + 2) / 3;
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x, nth = blockDim.x, E = A.E, tile = blockIdx.x;
  const LawP& L = A.law;
  const int epi = A.epi;
  // the state, aux and accumulators below may come from the previous kernel
  // of the stream (programmatic dependent launch, launch_maybe_pdl)
  pdl_wait();
  const int ne = min(E, A.K - tile * E);
  const size_t g0 = (size_t)tile * E * NP, stride = A.stride;
  // ---------------------------------------------------- this thread's line
  const int nld = E * NFP;
  const int d = (tid >= nld) + (tid >= 2 * nld);
  const int es_ = (tid - d * nld) / NFP;
  const bool line = es_ < ne && tid < 3 * nld;
  const int es = line ? es_ : 0;  // a thread without a line works on the first element and stores nothing
  const int l = tid < 3 * nld ? tid - d * nld - es_ * NFP : 0;
  const int e = tile * E + es;
  const bool act = (A.dirs >> d) & 1;
  double* const sq = sm + es * slotsz;
  double* const sx = sq + OX;
  const int base = line_base<NQ, 3>(d, l, ROW), sd = line_stride<NQ, 3>(d, ROW);
  // its two faces' neighbour nodes
  int nb[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) nb[i] = A.fnb[((size_t)e * 6 + 2 * d + i) * NFP + l];
  // --------------------------------------------------------- point values
  double qp[2][NS], ap[2];
  {
    double q[RN][NS], al[RN][3], mj[RN], g[RN][9];
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const int v = tid + r * nth;
      if (v < ne * NP) {
#pragma unroll
        for (int s = 0; s < NS; ++s) q[r][s] = A.q[s][g0 + v];
        al[r][0] = EG ? A.aux[g0 + v] : 0.0;
        if constexpr (FUSE) {
          al[r][1] = A.aux[4 * stride + g0 + v];
          al[r][2] = A.aux[5 * stride + g0 + v];
        }
        mj[r] = A.MJn[g0 + v];
#pragma unroll
        for (int k = 0; k < 9; ++k) g[r][k] = A.G[(size_t)k * stride + g0 + v];
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const size_t nid = nb[i] >= 0 ? (size_t)nb[i] : (size_t)e * NP;
#pragma unroll
      for (int s = 0; s < NS; ++s) qp[i][s] = A.q[s][nid];
      ap[i] = EG ? A.aux[nid] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const unsigned v = tid + r * nth;
      if (v < ne * NP) {
        const unsigned en = v / NP, n = v - en * NP;
        double* const so = sm + en * slotsz + n + (ROW - NQ) * (n / NQ);
        double* const xo = so + OX;
        const double rinv = rcp_cheb(q[r][0]);
        double u[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) u[c] = __dmul_rn(q[r][1 + c], rinv);
        double t = fma(-0.5, dot<3>(q[r] + 1, u), q[r][4]);
        if constexpr (EG) t = fma(-q[r][0], al[r][0], t);
        const double p = __dmul_rn(L.gamma - 1.0, t);
#pragma unroll
        for (int s = 0; s < NS; ++s) so[s * NPL] = q[r][s];
#pragma unroll
        for (int c = 0; c < 3; ++c) xo[c * NPL] = 0.5 * u[c];
        if constexpr (VK == VK_KG) {
          xo[3 * NPL] = 0.5 * p;
          xo[5 * NPL] = 0.5 * (q[r][4] * rinv);
        } else {
          const double pr = __dmul_rn(p, rinv);
          xo[3 * NPL] = rcp_cheb(pr);
          xo[5 * NPL] = pr;
        }
        xo[4 * NPL] = 0.25 * al[r][0];
#pragma unroll
        for (int k = 0; k < 9; ++k) xo[(CFD_NP + k) * NPL] = __dmul_rn(mj[r], g[r][k]);
        if constexpr (FUSE) {
          double pr;
          so[OL] = __dmul_rn(A.lin_law.gamma - 1.0, fma(-q[r][0], al[r][0], q[r][4]));
          so[OL + NPL] = lin_enthalpy(A.lin_gg1, al[r][0], al[r][1], al[r][2], &pr);
        }
      }
    }
  }
  __syncthreads();
  // ------------------------------------------------------ the line's sums
  double fm[2], nrm[2][3];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const size_t fj = ((size_t)e * 6 + 2 * d + i) * NFP + l;
#pragma unroll
    for (int c = 0; c < 3; ++c) nrm[i][c] = A.fnrm[fj * 3 + c];
    fm[i] = A.fMJ[fj];
  }
  if constexpr (FUSE) {
    // the weak-form linear operator along the radial lines: D^T of the
    // contravariant rows [U, p' l, H U] (U = l . rho u), the faces
    if (d == 2 && line) {
      double t[NQ][NS];
#pragma unroll
      for (int a = 0; a < NQ; ++a)
#pragma unroll
        for (int s = 0; s < NS; ++s) t[a][s] = 0.0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int nm = base + (i ? (NQ - 1) * sd : 0);
        const size_t mid = (size_t)e * NP + l + (i ? (NQ - 1) * NFP : 0), nid = nb[i] >= 0 ? (size_t)nb[i] : mid;
        double qm[NS], qb[NS], nf[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          qm[s] = sq[s * NPL + nm];
          qb[s] = qp[i][s];
        }
        double Pb = ap[i];
        if (nb[i] < 0) {
          boundary_state_n(A.lin_law, nrm[i], -1 - nb[i], qm, qb);
          Pb = 4.0 * sx[4 * NPL + nm];
        }
        double prm, prp;
        lin_enthalpy(A.lin_gg1, 0.0, A.aux[4 * stride + mid], A.aux[5 * stride + mid], &prm);
        const double Hp = lin_enthalpy(A.lin_gg1, Pb, A.aux[4 * stride + nid], A.aux[5 * stride + nid], &prp);
        const double pl = __dmul_rn(A.lin_law.gamma - 1.0, fma(-qb[0], Pb, qb[4]));
        const double mm = dot<3>(qm + 1, nrm[i]), mp = dot<3>(qb + 1, nrm[i]);
        // max(sqrt a, sqrt b) = sqrt(max(a, b))
        const double ws = -0.5 * sqrt_house(__dmul_rn(A.lin_law.gamma, dmax(prm, prp)));
        const double ps = 0.5 * (sq[OL + nm] + pl);
        nf[0] = fma(ws, qb[0] - qm[0], 0.5 * (mm + mp));
#pragma unroll
        for (int c = 0; c < 3; ++c) nf[1 + c] = fma(ws, qb[1 + c] - qm[1 + c], __dmul_rn(ps, nrm[i][c]));
        nf[4] = fma(ws, qb[4] - qm[4], 0.5 * fma(Hp, mp, __dmul_rn(sq[OL + NPL + nm], mm)));
#pragma unroll
        for (int s = 0; s < NS; ++s) t[i ? NQ - 1 : 0][s] = __dmul_rn(-fm[i], nf[s]);
      }
#pragma unroll
      for (int m = 0; m < NQ; ++m) {
        const int n = base + m * sd;
        double lv[3], mo[3], row[NS];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          lv[c] = sx[(CFD_NP + 6 + c) * NPL + n];
          mo[c] = sq[(1 + c) * NPL + n];
        }
        row[0] = dot<3>(lv, mo);
#pragma unroll
        for (int c = 0; c < 3; ++c) row[1 + c] = __dmul_rn(sq[OL + n], lv[c]);
        row[4] = __dmul_rn(sq[OL + NPL + n], row[0]);
#pragma unroll
        for (int a = 0; a < NQ; ++a)
#pragma unroll
          for (int s = 0; s < NS; ++s) t[a][s] = fma(A.cfd[m * NQ + a], row[s], t[a][s]);
      }
#pragma unroll
      for (int a = 0; a < NQ; ++a)
#pragma unroll
        for (int s = 0; s < NS; ++s) sq[OT + s * NPL + base + a * sd] = t[a][s];
    }
  }
  double T[NQ][NS];
#pragma unroll
  for (int a = 0; a < NQ; ++a)
#pragma unroll
    for (int s = 0; s < NS; ++s) T[a][s] = 0.0;
  if (act) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int nm = base + (i ? (NQ - 1) * sd : 0);
      const size_t mid = (size_t)e * NP + line_base<NQ, 3>(d, l, NQ) + (size_t)(i ? NQ - 1 : 0) * line_stride<NQ, 3>(d, NQ);
      double qm[NS], qb[NS], nf[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        qm[s] = sq[s * NPL + nm];
        qb[s] = qp[i][s];
      }
      const double Pm = EG ? 4.0 * sx[4 * NPL + nm] : 0.0;
      double Pb = ap[i];
      if (nb[i] < 0) {
        boundary_state_n(L, nrm[i], -1 - nb[i], qm, qb);
        Pb = Pm;
      }
      if constexpr (SF == F_RUSANOV) {
        double dm = 0.0, dp = 0.0;
        if (EG && L.pde) {  // pde_level_balance
          dm = A.aux[5 * stride + mid];
          dp = nb[i] >= 0 ? A.aux[5 * stride + nb[i]] : dm;
        }
        curved_rusanov<LAW>(L, nrm[i], qm, Pm, dm, qb, Pb, dp, nf);
      } else {
        double am[NA], av[NA];
#pragma unroll
        for (int k = 0; k < NA; ++k) {
          am[k] = k < A.naux_nl ? A.aux[(size_t)k * stride + mid] : 0.0;
          av[k] = k < A.naux_nl && nb[i] >= 0 ? A.aux[(size_t)k * stride + nb[i]] : am[k];
        }
        curved_flux_any<LAW>(L, A.sflux, nrm[i], qm, am, qb, av, nf);
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) T[i ? NQ - 1 : 0][s] = __dmul_rn(-fm[i], nf[s]);
    }
  }
  if (act) {
    if constexpr (VK == VK_EC) {
      // the form of the line's logarithmic means (atb_fd.cuh)
      int rlo = 0x7fffffff, rhi = -0x7fffffff - 1, blo = rlo, bhi = rhi;
#pragma unroll
      for (int a = 0; a < NQ; ++a) {
        const int hr = __double2hiint(sq[base + a * sd]), hb = __double2hiint(sx[3 * NPL + base + a * sd]);
        rlo = min(rlo, hr);
        rhi = max(rhi, hr);
        blo = min(blo, hb);
        bhi = max(bhi, hb);
      }
      const double rmax = __hiloint2double(rhi + 1, 0), bmax = __hiloint2double(bhi + 1, 0);
      const double rmin = __hiloint2double(rlo, 0), bmin = __hiloint2double(blo, 0);
      const double c0 = 2.0 / (L.gamma - 1.0);
      const bool plain = min(rlo, blo) >= ((1023 - 240) << 20) && max(rhi, bhi) < ((1023 + 240) << 20);
      if (plain && rmax < 1.2 * rmin && bmax < 1.2 * bmin)
        curved_pairs<LAW, VK, NQ, 0>(A, c0, sq, sx, base, sd, d, T);
      else if (plain && rmax < 3.0 * rmin && bmax < 3.0 * bmin)
        curved_pairs<LAW, VK, NQ, 1>(A, c0, sq, sx, base, sd, d, T);
      else
        curved_pairs<LAW, VK, NQ, 2>(A, c0, sq, sx, base, sd, d, T);
    } else {
      curved_pairs<LAW, VK, NQ, 0>(A, 0.0, sq, sx, base, sd, d, T);
    }
  }
  __syncthreads();  // the point values are dead: their region takes the sums
  if (line) {
#pragma unroll
    for (int a = 0; a < NQ; ++a)
#pragma unroll
      for (int s = 0; s < NS; ++s) sx[(d * NS + s) * NPL + base + a * sd] = T[a][s];
  }
  __syncthreads();
  // ------------------------------------------------------------- epilogue
  const bool cor = L.src == SRC_CORIOLIS && ((A.dirs >> 2) & 1);
#pragma unroll 1
  for (int v = tid; v < ne * NP; v += nth) {
    const unsigned en = (unsigned)v / NP, n = v - en * NP;
    const double* const qn = sm + en * slotsz + n + (ROW - NQ) * (n / NQ);
    const size_t gid = g0 + v;
    const double mji = rcp_cheb(A.MJn[gid]);
    double t[NS], tl[NS], in[2][NS], gp[3];
    const bool rd = FUSE || epi == EPI_ADD || (epi == EPI_LSRK && A.a != 0.0) || epi == EPI_SUBOUT2 || epi == EPI_RLSRK;
    const bool o2 = epi == EPI_SUBOUT2 || epi == EPI_RLSRK;
    if (rd) {
#pragma unroll
      for (int i = 0; i < (FUSE ? 2 : 1); ++i)
        if (!FUSE || A.accin[i][0]) {
#pragma unroll
          for (int s = 0; s < NS; ++s) in[i][s] = (FUSE ? A.accin[i][s] : o2 ? A.out2[s] : A.out[s])[gid];
        }
    }
    if constexpr (FUSE) {
#pragma unroll
      for (int k = 0; k < 3; ++k) gp[k] = A.aux[(1 + k) * stride + gid];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) t[s] = __dmul_rn(mji, (qn[OX + s * NPL] + qn[OX + (NS + s) * NPL]) + qn[OX + (2 * NS + s) * NPL]);
    auto coriolis = [&](const double* om, double* w) {
      const double m0 = qn[NPL], m1 = qn[2 * NPL], m2 = qn[3 * NPL];
      w[1] -= fma(om[1], m2, -__dmul_rn(om[2], m1));
      w[2] -= fma(om[2], m0, -__dmul_rn(om[0], m2));
      w[3] -= fma(om[0], m1, -__dmul_rn(om[1], m0));
    };
    if (cor) coriolis(L.omega, t);
    if constexpr (FUSE) {
#pragma unroll
      for (int s = 0; s < NS; ++s) tl[s] = __dmul_rn(mji, qn[OT + s * NPL]);
#pragma unroll
      for (int k = 0; k < 3; ++k) tl[1 + k] = fma(-qn[0], gp[k], tl[1 + k]);
      if (A.lin_law.src == SRC_CORIOLIS) coriolis(A.lin_law.omega, tl);
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (A.acc[j][0]) {
          const bool r2 = A.accin[j][0] != nullptr;  // accumulators read and written come first (run_fused)
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const double b = r2 ? in[j < 2 ? j : 1][s] : qn[s * NPL];
            A.acc[j][s][gid] = fma(A.adt, fma(A.ca[j], t[s] - tl[s], __dmul_rn(A.cb[j], tl[s])), b);
          }
        }
    } else if (epi == EPI_LSRK) {
      const double bdt = A.dte ? A.bdt * A.dte[tile * E + en] : A.bdt;
      if (A.a != 0.0) {
#pragma unroll
        for (int s = 0; s < NS; ++s) t[s] = fma(A.a, in[0][s], t[s]);
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        A.out[s][gid] = t[s];
        A.out2[s][gid] = fma(bdt, t[s], qn[s * NPL]);
      }
    } else if (epi == EPI_SET) {
#pragma unroll
      for (int s = 0; s < NS; ++s) A.out[s][gid] = t[s];
    } else if (epi == EPI_ADD) {
#pragma unroll
      for (int s = 0; s < NS; ++s) A.out[s][gid] = in[0][s] + t[s];
    } else if (epi == EPI_SUBOUT2) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        A.out[s][gid] = t[s];
        A.out2[s][gid] = in[0][s] - t[s];
      }
    } else if (epi == EPI_RLSRK) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        A.out[s][gid] = t[s];
        A.out2[s][gid] = fma(A.a, in[0][s], t[s]);
      }
    } else {  // EPI_ARK after a separate explicit launch: out holds N(Q), t = L(Q)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (A.acc[j][0]) {
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const double b = A.accin[j][0] ? A.accin[j][s][gid] : qn[s * NPL];
            A.acc[j][s][gid] = b + A.adt * (A.ca[j] * (A.out[s][gid] - t[s]) + A.cb[j] * t[s]);
          }
        }
    }
  }
  pdl_trigger();
}

template <int LAW, int VK, int NQ, bool FUSE, int SF>
void curved_fd_launch(const TendArgs& A, int grid, int block, size_t smem, cudaStream_t st) {
  static SmemLimit limit;
  raise_smem(curved_fd_kernel<LAW, VK, NQ, FUSE, SF>, limit, smem);
  launch_maybe_pdl(curved_fd_kernel<LAW, VK, NQ, FUSE, SF>, dim3(grid), dim3(block), smem, st, A);
}

template <int LAW, int VK, bool FUSE, int SF> tend_launch_fn curved_fd_pick(int nq) {
  switch (nq) {
    case 2: return curved_fd_launch<LAW, VK, 2, FUSE, SF>;
    case 3: return curved_fd_launch<LAW, VK, 3, FUSE, SF>;
    case 4: return curved_fd_launch<LAW, VK, 4, FUSE, SF>;
    case 5: return curved_fd_launch<LAW, VK, 5, FUSE, SF>;
    case 6: return curved_fd_launch<LAW, VK, 6, FUSE, SF>;
    case 7: return curved_fd_launch<LAW, VK, 7, FUSE, SF>;
    case 8: return curved_fd_launch<LAW, VK, 8, FUSE, SF>;
  }
  return nullptr;
}

}  // namespace atb
