// Flux-differencing tendency kernel, one thread per tensor line.  (Measured on
// B200 against the node-per-thread form that stored every pair in shared
// memory: 16^3 elements at N = 4, fused ARK23 stage 88 -> 52 us by events around
// each launch (80 -> 44 by difference from the step); 32^3 at N = 7, 5.11 -> 1.66 ms; 128 shallow-water basins of 32^2 at N = 4, FP32
// flux, 267 -> 114 us per LSRK stage; weak form, 24^3 at N = 4: 206 -> 76 us.)
//
// The same stage as atb_tendency.cuh's kernel (volume term, surface term,
// sources, the stepper's write-back; the fused ARK23 stage with the weak-form
// linear operator along z), for the two-point volume fluxes and the weak form of
// 3-D Euler-gravity, at the compiled orders (2 <= Nq <= 8).
//
// What bounds it: the FP64 pipe (64 lanes per SM: one warp instruction per two
// cycles and scheduler) and, around it, the latency of the staging loads.  The
// two-point flux of a node pair is symmetric, so a thread owns one line of Nq
// nodes in one direction: it reads each node's point values from shared memory,
// evaluates every unordered pair of the line once and adds it to both nodes'
// accumulators in registers.  Nothing per pair goes through shared memory (the
// node-per-thread form stored NS + 1 values per pair and read them back twice)
// and the pairs of a line are independent, so the FP64 latency is covered by
// the pairs of one thread as well as by the warps.  Dim * Nq^(dim-1) lines per
// element run in parallel; afterwards the directions add their accumulators
// into one shared array in turn (fixed order: results do not depend on the
// launch shape).
//
// Direction-agnostic code: a thread reads the velocity (momentum) components
// rotated so that its line's normal component comes first, so one instruction
// stream serves all directions, lanes of one warp included.  The FP32-flux
// entropy-conservative flux keeps the components in x, y, z order and selects
// (its FP32 sums then round as they always did).
//
// Shared memory per element: state (NS), point values (NX), all in rows of
// Nq | 1 doubles (an odd row stride keeps x-lines free of bank conflicts); the
// accumulators reuse the point values' region after the volume term.
#pragma once
#include "atb_tendency.cuh"

#include <type_traits>

namespace atb {

// sqrt(x) for x = 0 and normal x: the hardware's reciprocal square root y0 (relative
// error <= 2^-20), one third-order Householder step y = y0 (1 + e/2 + 3 e^2/8),
// e = 1 - x y0^2, then one Heron correction of s = x y: 0.51 ulp from 2^-968 on
// (0.64 below, where the correction's residual underflows; tests/test_elementary.py).
// NaN for negative, subnormal and infinite x.
__device__ __forceinline__ double sqrt_house(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-__dmul_rn(x, y), y, 1.0);
  y = fma(__dmul_rn(y, e), fma(0.375, e, 0.5), y);
  const double s = __dmul_rn(x, y);
  const double t = fma(__dmul_rn(0.5, y), fma(-s, s, x), s);
  return x == 0.0 ? x : t;
}

template <int LAW, int DIM, int VK> struct LineShape {
  static constexpr int NS = NSt<LAW, DIM>::v;
  static constexpr bool EG = LAW == LAW_EG;
  static constexpr bool SW = LAW == LAW_SW;
  static constexpr bool F32 = VK == VK_EC32 || VK == VK_KG32;
  // a third quantity per node pair, contracted like the flux and scaled by a
  // node value at the end: the gravity fluctuation (EG) or the bathymetry
  // difference (shallow water)
  static constexpr bool XTRA = (EG || SW) && VK != VK_WEAK;
  // point values per node, in doubles:
  //   EC (Euler, EG)  u/2 (DIM), B = rho/p, p/rho [, Phi/4]
  //   KG              u/2 (DIM), p/2, e/2 [, Phi/4]
  //   EC32            p, b = rho/2p, p/rho [, Phi], then FP32 u (DIM), |u|^2
  //   KG32            p [, Phi], then FP32 u (DIM), e
  //   WEAK (EG)       1/rho, p (less the reference), rho e + p, Phi/4
  //   EC (SW)         u/2 (DIM), theta/2, b
  //   EC32 (SW)       b, then FP32 u (DIM), theta
  static constexpr int ND = VK == VK_WEAK ? 4
                               : SW ? (F32 ? 1 : DIM + 2)
                               : (VK == VK_EC32) ? 3 + (EG ? 1 : 0) : (VK == VK_KG32) ? 1 + (EG ? 1 : 0)
                                                                                       : DIM + 2 + (EG ? 1 : 0);
  static constexpr int NF = F32 ? DIM + 1 : 0;  // FP32 values
  static constexpr int NX = ND + (NF + 1) / 2;
  // the accumulators (NS per node) reuse the region of the point values
  static constexpr int NXA = NX > NS ? NX : NS;
};

__host__ __device__ constexpr int line_row(int nq) { return nq | 1; }
__host__ __device__ constexpr int line_nodes(int nq, int dim) { return line_row(nq) * ipow(nq, dim - 1); }
// Per kernel: the largest CTA it is compiled for (every line of a CTA's
// elements has its own thread), the resident CTAs the register budget is set
// for, and the accumulator arrays in shared memory: one per direction (every
// direction writes its own, one barrier) or one that the directions add into in
// turn.  Measured per order on B200: more warps pay until the spills they force
// cost more (3-D, Nq = 6: 718 us per LSRK54 step of 20^3 elements at 4 CTAs of
// 128 threads, 750 at 2 of 224; Nq = 5 fused stage, by difference
// from the step: 44 us at 3 CTAs of 160 threads, 49 at 2, 74 at 4); one accumulator array pays where shared memory
// or the FP32-flux form's registers limit the CTAs (shallow water, Nq = 5:
// 561 against 612 us).
struct FdCfg {
  int max_threads, min_blocks, bufs;
};
__host__ __device__ constexpr FdCfg fd_cfg(int law, int dim, int vk, int nq) {
  const bool f32 = vk == VK_EC32 || vk == VK_KG32;
  if (dim == 2 && law == LAW_SW) return FdCfg{160, nq <= 5 ? 4 : 3, 1};
  // (Nq = 4, FP64: 136 registers without a bound, two CTAs all the same; held to 128 it
  // spills, 8x8 elements at 10 LSRK54 steps 173 -> 179 us)
  if (dim == 2) return FdCfg{224, nq == 4 && vk == VK_EC ? 1 : 2, 2};
  // weak form: little arithmetic, so more CTAs for the memory (24^3 elements, N =
  // 4: 75 us at 4 of 160 threads and one array, 82 at 3 and three arrays, 95 at
  // 8 of 96, 102 at 5 of 160; N = 1: 109 us at 8 of 96, 132 at 4 of 160)
  if (vk == VK_WEAK && nq <= 5) return nq == 2 ? FdCfg{96, 8, 1} : FdCfg{160, 4, 1};
  if (nq == 8) return FdCfg{192, 2, 1};
  if (nq == 7) return FdCfg{160, 3, 1};
  if (nq == 6) return FdCfg{128, 4, 1};
  if (nq == 5 || f32) return FdCfg{160, 3, f32 ? 1 : 3};
  // (Nq = 4, FP64 EC: 147 registers and no spill; held to 128, ARK23 steps of 13x16x4
  // elements take 36.7 us instead of 35.1)
  return FdCfg{224, nq == 4 && vk == VK_EC ? 1 : 2, 3};
}
__host__ __device__ constexpr int line_count(int nq, int dim) { return dim * ipow(nq, dim - 1); }
inline int fd_max_elements(int law, int dim, int vk, int nq) {
  const int m = fd_cfg(law, dim, vk, nq).max_threads / line_count(nq, dim);
  return m < 1 ? 1 : m;
}
// Elements per CTA when nothing else asks for a count: the fullest last warp
// among CTAs of at least 96 threads (the smallest such), but no fewer CTAs than
// SMs where the operator has the elements for it.  While every element's warps
// can have a scheduler to themselves, one element: the pairs take as long as in
// a full warp and the other lanes share the staging (2-D Euler-gravity N = 7,
// 24x24 elements: 10.2 us per LSRK54 stage at 4 elements, 9.0 at 1; 3-D N = 3,
// 6^3: 4.1 at 2, 3.6 at 1); not below 16 lines an element, where it measured
// within 4 % either way, on curved elements (162 at N = 4: 8.4 us at 2, 8.9 at 1), or
// where the FP32 surface flux is chosen at run time (a copy per direction, which
// warps of one direction run alone: 6^3 at N = 3, 6.4 us at 2, 8.0 at 1).
inline int fd_default_elements(int nq, int dim, int emax, int K, int nsm, bool one) {
  const int nl = line_count(nq, dim);
  if (one && nq >= 4 && nl >= 16 && (long long)K * ((nl + 31) / 32) <= 4LL * nsm) return 1;
  int best = emax;
  double fill = 0.0;
  for (int E = 1; E <= emax; ++E) {
    const int th = ((E * nl + 31) / 32) * 32;
    if (th < 96 && E < emax) continue;
    const double f = (double)(E * nl) / th;
    if (f > fill + 1e-9) { fill = f; best = E; }
  }
  const int spread = (K + nsm - 1) / nsm;
  return best < spread ? best : spread < 1 ? 1 : spread;
}
inline int fd_threads(int nq, int dim, int E) { return ((E * line_count(nq, dim) + 31) / 32) * 32; }
// doubles per element; nxa: point values per node (fd_nx)
__host__ __device__ constexpr int fd_slot(int ns, int nxa, int nq, int dim, int bufs, bool fuse) {
  const int npl = line_nodes(nq, dim);
  // fused: linear p' and (rho e + p)_ref / rho_ref * m_z, the linear tendency
  return (ns + nxa + (fuse ? 2 + ns : 0) + (bufs - 1) * ns) * npl;
}
inline int fd_nx(int law, int dim, int vk) {
  const int ns = dim + 2;
  const bool f32 = vk == VK_EC32 || vk == VK_KG32;
  const int eg = law == LAW_EG ? 1 : 0;
  const int nd = vk == VK_WEAK ? 4 : law == LAW_SW ? (f32 ? 1 : dim + 2) : vk == VK_EC32 ? 3 + eg : vk == VK_KG32 ? 1 + eg : dim + 2 + eg;
  const int nx = nd + (f32 ? (dim + 2) / 2 : 0);
  return nx > ns ? nx : ns;
}
inline size_t fd_smem_bytes(int law, int dim, int vk, int nq, int E, bool fuse) {
  const int slot = fd_slot(dim + 2, fd_nx(law, dim, vk), nq, dim, fd_cfg(law, dim, vk, nq).bufs, fuse);
  return sizeof(double) * ((size_t)nq * nq + 2 + (size_t)E * slot);
}

// ---------------------------------------------------- grids of one wave
// A line's thread evaluates its pairs one after the other, 28 at Nq = 8, and both
// face fluxes: where the whole grid is resident at once, a launch takes as long as
// that chain.  The SMALL mode of the kernel has one element per CTA and spreads
// the pairs and the faces of its lines over all threads, values through shared
// memory; the node's thread sums them in the order of the line's thread.  The same
// operations on the same values give the same bits, so the mode may be chosen by
// the element count.  us per LSRK54 stage, line per thread / SMALL:
//   2-D Euler-gravity FP64 N = 7, 8x8 elements 7.9 / 4.9, 24x24 8.8 / 7.1 (96
//   threads; 10.2 with 448), 40x40 11.6 / 16.7; FP32 flux 8x8 11.6 / 5.6, 32x32
//   15.1 / 11.9; Roe flux 8x8 11.5 / 6.8; 2-D Euler FP64 N = 5, 8x8 5.1 / 4.3,
//   N = 4 3.7 / 4.3.  3-D: FP64 pairs gain nothing (N = 4, 27 elements 4.9 / 5.6);
//   FP32-flux EC, ARK23 step, 3^3 N = 4 51 / 33, N = 6 95 / 56, 6^3 N = 7 112 /
//   149; weak form with Roe's flux, 5^3 N = 4 9.3 / 6.9.
__host__ __device__ constexpr int small_pairs(int nq) { return nq * (nq - 1) / 2; }
// directions whose pairs share the buffer: all, while they leave room for two CTAs
__host__ __device__ constexpr int small_batch(int nq, int dim) { return dim == 2 || nq <= 6 ? dim : 1; }
// a thread for every node and face, the most for the pairs
__host__ __device__ constexpr int small_least(int nq, int dim) {
  const int faces = 2 * line_count(nq, dim), nodes = ipow(nq, dim);
  return ((faces > nodes ? faces : nodes) + 31) / 32 * 32;
}
__host__ __device__ constexpr int small_threads(int nq, int dim) {
  const int pairs = (line_count(nq, dim) * small_pairs(nq) + 31) / 32 * 32;
  const int cap = dim == 2 ? 448 : nq <= 5 ? 288 : nq == 6 ? 384 : 512;
  const int most = pairs < cap ? pairs : cap;
  return most > small_least(nq, dim) ? most : small_least(nq, dim);
}
// where it is compiled (sf < 0: the surface flux chosen at run time)
__host__ __device__ constexpr bool fd_has_small(int law, int dim, int vk, int sf) {
  if (dim == 2) return law == LAW_EULER || law == LAW_EG;
  return law == LAW_EG && (vk == VK_EC32 || (vk == VK_WEAK && sf < 0));
}
// Threads per CTA of the SMALL mode, 0 where a thread per line is faster (measured
// per order; K elements, nsm multiprocessors): 2-D up to four elements per
// multiprocessor, where FP64 pairs with Rusanov's flux are many (Nq >= 6) or the
// chain is long otherwise (Nq >= 4), and seven for the longest; 3-D one, or as far
// as its CTAs are resident together.  Fewer threads as the elements get more.
inline int fd_small(int law, int dim, int vk, int nq, int sf, int K, int nsm) {
  const bool any = sf != F_RUSANOV;
  if (!fd_has_small(law, dim, vk, any ? -1 : sf)) return 0;
  const bool slow = vk == VK_EC32 || any;
  int most = 0;  // elements per two multiprocessors
  if (dim == 2)
    most = nq == 8 && slow ? 14 : nq >= 6 || (slow && nq >= 4) ? 8 : 0;
  else if (vk == VK_WEAK)
    most = nq == 4 ? 8 : nq == 5 || nq == 6 ? 3 : nq == 7 ? 2 : 0;
  else
    most = nq >= 4 && nq <= 7 ? 2 : 0;
  if (2LL * K > (long long)most * nsm) return 0;
  const int cap = K <= nsm ? small_threads(nq, dim) : K <= 4 * nsm ? 96 : 64;
  const int least = small_least(nq, dim), full = small_threads(nq, dim);
  const int t = cap < full ? cap : full;
  return t > least ? t : least;
}
// doubles of shared memory: tables, the element, face fluxes, line forms and pair
// numbers, pair values (NS and the extra one)
__host__ __device__ constexpr int small_slot(int ns, int nxa, int nq, int dim, bool fuse) {
  return (ns + nxa + (fuse ? 2 + ns : 0)) * line_nodes(nq, dim);
}
__host__ __device__ constexpr int small_doubles(int ns, int nxa, int nq, int dim, bool fuse, bool pairs) {
  const int nl = line_count(nq, dim), np = small_pairs(nq);
  return 2 * nq * nq + 2 + small_slot(ns, nxa, nq, dim, fuse) + 2 * nl * ns + (nl + np + 1) / 2 +
         (pairs ? small_batch(nq, dim) * ipow(nq, dim - 1) * np * (ns + 1) : 0);
}

// ------------------------------------------------------------ pair fluxes
// Point values of one node as a pair flux reads them; velocities rotated
// (normal component first) in the FP64 forms.
template <int LAW, int DIM, int VK> struct LinePt {
  double r, v[DIM + 1], ph;     // EC: v = u/2 .., B; KG: u/2 .., e/2; SW: u/2 .., theta/2
  double w;                     // KG: p/2; SW: normal momentum / 2
  double p, b;                  // EC32: p, b; KG32: p
  float uf[DIM], xf;            // EC32: u, |u|^2; KG32: u, e; SW EC32: u, theta
};

// VOL: read again for every pair (volatile): at Nq >= 6 in 3-D the compiler
// would keep a line's values in registers it does not have, and spill (Nq = 8:
// 1663 -> 1624 us per ARK23 step of 20^3 elements, Nq = 7: 1026 -> 970)
template <int LAW, int DIM, int VK, bool VOL>
__device__ __forceinline__ void line_load(LinePt<LAW, DIM, VK>& P, const double* sq_, const double* sx_, int npl, int n,
                                          const int* rot, int d) {
  using S = LineShape<LAW, DIM, VK>;
  using Ptr = std::conditional_t<VOL, const volatile double*, const double*>;
  using FPtr = std::conditional_t<VOL, const volatile float*, const float*>;
  const Ptr sq = sq_, sx = sx_;
  P.r = sq[n];
  if constexpr (S::SW) {
    P.w = sq[(1 + d) * npl + n];
    P.ph = sx[(S::ND - 1) * npl + n];
    if constexpr (S::F32) {
      const FPtr sf = (const float*)(sx_ + S::ND * npl);
#pragma unroll
      for (int c = 0; c < DIM; ++c) P.uf[c] = sf[rot[c] * npl + n];
      P.xf = sf[DIM * npl + n];
    } else {
#pragma unroll
      for (int c = 0; c < DIM; ++c) P.v[c] = sx[rot[c] * npl + n];
      P.v[DIM] = sx[DIM * npl + n];
    }
  } else if constexpr (S::F32) {
    P.p = sx[n];
    if constexpr (VK == VK_EC32) P.b = sx[npl + n];
    if constexpr (S::EG) P.ph = sx[(S::ND - 1) * npl + n];
    const FPtr sf = (const float*)(sx_ + S::ND * npl);
#pragma unroll
    for (int c = 0; c < DIM; ++c) P.uf[c] = sf[(VK == VK_KG32 ? rot[c] : c) * npl + n];
    P.xf = sf[DIM * npl + n];
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) P.v[c] = sx[rot[c] * npl + n];
    if constexpr (VK == VK_KG) {
      P.w = sx[DIM * npl + n];
      P.v[DIM] = sx[(DIM + 1) * npl + n];
    } else {
      P.v[DIM] = sx[DIM * npl + n];
    }
    if constexpr (S::EG) P.ph = sx[(S::ND - 1) * npl + n];
  }
}

// The FP32-flux EC pair of ec_vol32 for a line whose values lie within a factor 1.2
// (both logarithmic means on their series branch): the same FP32 operations and
// roundings without a branch, a call or a division, so that a line's pairs overlap;
// the quotients of one divisor share its reciprocal.  (2-D Euler N = 7, 24x24
// elements: 18.3 -> 11.1 us per LSRK54 stage; 3-D Euler-gravity N = 5, 10^3: 30.7 ->
// 25.3.  What is left is conversions, 14 or 15 a pair.)
template <int LAW, int DIM>
__device__ __forceinline__ void ec_line32(float igm1, int d, const LinePt<LAW, DIM, VK_EC32>& P,
                                          const LinePt<LAW, DIM, VK_EC32>& Q, double* f, double* xtra) {
  const double rs64 = P.r + Q.r, bs64 = P.b + Q.b;
  const double rho_avg = rs64 * 0.5, p_avg = (P.p + Q.p) * 0.5;
  const float rs = (float)rs64, rd = (float)(P.r - Q.r), bs = (float)bs64, bd = (float)(P.b - Q.b);
  const float ir = rcp32(rs), ib = rcp32(bs);
  const float fr = div32(rd, rs, ir), fb = div32(bd, bs, ib);
  const float ur = fr * fr, ub = fb * fb;
  const float cr = ur * (1.f / 3.f + ur * (4.f / 45.f + ur * (44.f / 945.f + ur * (428.f / 14175.f +
                   ur * (10196.f / 467775.f + ur * (10719068.f / 638512875.f + ur * (25865068.f / 1915538625.f)))))));
  const double rho_log = rho_avg - rho_avg * (double)cr;
  const float cterm = div32(series_F(ub) * igm1, bs, ib);
  const double corr = (double)div32((float)(P.p - Q.p) * -bd, 2.f * bs, 0.5f * ib);
  const double pc = p_avg - corr;
  float ua[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) ua[c] = 0.5f * (P.uf[c] + Q.uf[c]);
  const float rl = (float)rho_log;
  float ud = ua[0];
#pragma unroll
  for (int c = 1; c < DIM; ++c)
    if (c == d) ud = ua[c];
  const float frd = ud * rl;
  f[0] = (double)frd;
  float mu = 0.f;
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const float m = ud * (ua[c] * rl);
    f[1 + c] = (double)m;
    mu += m * ua[c];
  }
#pragma unroll
  for (int c = 0; c < DIM; ++c)
    if (c == d) f[1 + c] += pc;
  mu += (float)pc * ud;
  float c1 = cterm - 0.25f * (P.xf + Q.xf);
  if (LAW == LAW_EG) c1 += (float)((P.ph + Q.ph) * 0.5);
  f[DIM + 1] = (double)(c1 * frd + mu);
  *xtra = (bs64 * 0.5) * rho_log;
}

// Symmetric two-point flux f (components rotated: normal momentum at 1, except
// VK_EC32, x y z order) and the extra value x, antisymmetric in the pair.
//   EC: rho_log, p_c = rho_avg / (2 b_avg), and the energy flux in the form
//       f_rho (1/(2 (g-1) b_log) + Phi_avg + u1.u2 / 2) + p_c u_n
//       (|u_avg|^2 - |u|^2_avg / 2 = u1.u2 / 2), with one reciprocal for every
//       division: B = rho/p, R = rho_1 + rho_2, S = B_1 + B_2,
//       p_c = R/S, 1/(2 (g-1) b_log) = 2 F(u_B) / ((g-1) S).
//   TIER: the line's values lie within a factor 1.2 (0), within a factor 3 (1: a
//   longer polynomial; the core of a vortex on a coarse grid), or further apart
//   (2: logarithms).  The form depends on the line alone, so results do not
//   depend on the launch shape.  FP32-flux form: 0 (ec_line32), or a branch per
//   pair (2), which gives near pairs the same values.
template <int LAW, int DIM, int VK, int TIER>
__device__ __forceinline__ void line_pair(const LawP& L, double c0, int d, const LinePt<LAW, DIM, VK>& P,
                                          const LinePt<LAW, DIM, VK>& Q, double* f, double& x) {
  using S = LineShape<LAW, DIM, VK>;
  if constexpr (S::SW && !S::F32) {
    const double md = 0.5 * (P.w + Q.w);
    f[0] = md;
#pragma unroll
    for (int c = 0; c < DIM; ++c) f[1 + c] = md * (P.v[c] + Q.v[c]);
    f[1] = fma(c0 * P.r, Q.r, f[1]);  // g h1 h2 / 2
    f[DIM + 1] = md * (P.v[DIM] + Q.v[DIM]);
    x = P.ph - Q.ph;
  } else if constexpr (S::SW) {
    const double md = 0.5 * (P.w + Q.w);
    const float mdf = (float)md;
    f[0] = md;
#pragma unroll
    for (int c = 0; c < DIM; ++c) f[1 + c] = (double)(mdf * (0.5f * (P.uf[c] + Q.uf[c])));
    f[1] += L.grav * P.r * Q.r * 0.5;
    f[DIM + 1] = (double)(mdf * (0.5f * (P.xf + Q.xf)));
    x = P.ph - Q.ph;
  } else if constexpr (VK == VK_KG32) {
    kg_vol32<DIM>(0, P.r, P.p, P.uf, P.xf, Q.r, Q.p, Q.uf, Q.xf, f);
    if constexpr (S::EG) x = ((P.r + Q.r) / 2.0 / 2.0) * (P.ph - Q.ph);
  } else if constexpr (VK == VK_EC32) {
    // ec_vol32 with the direction given at run time (the FP32 sums stay in
    // x, y, z order)
    double xr;
    if constexpr (TIER == 0)
      ec_line32<LAW, DIM>((float)c0, d, P, Q, f, &xr);
    else
      ec_vol32<LAW, DIM>((float)c0, d, P.r, P.p, P.b, P.uf, P.xf, S::EG ? P.ph : 0.0, Q.r, Q.p, Q.b, Q.uf, Q.xf,
                         S::EG ? Q.ph : 0.0, f, &xr);
    if constexpr (S::EG) x = xr * (P.ph - Q.ph);
  } else if constexpr (VK == VK_KG) {
    const double ravg = 0.5 * (P.r + Q.r);
    double ua[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) ua[c] = P.v[c] + Q.v[c];
    const double pa = P.w + Q.w, ea = P.v[DIM] + Q.v[DIM];
    const double fr = ua[0] * ravg;
    f[0] = fr;
#pragma unroll
    for (int c = 0; c < DIM; ++c) f[1 + c] = (c == 0) ? fma(fr, ua[c], pa) : fr * ua[c];
    f[DIM + 1] = fma(fr, ea, ua[0] * pa);
    if constexpr (S::EG) x = ravg * (2.0 * (P.ph - Q.ph));  // rho_avg / 2 (Phi1 - Phi2)
  } else {
    const double R = P.r + Q.r, rd = P.r - Q.r, B = P.v[DIM] + Q.v[DIM], bd = P.v[DIM] - Q.v[DIM];
    double rl, pc, ct;
    if constexpr (TIER < 2) {
      const double R2 = R * R, B2 = B * B;
      const double inv = rcp_cheb(R2 * B2);
      const double ib2 = R2 * inv, ir2 = B2 * inv;  // 1 / S^2, 1 / R^2
      const double iB = B * ib2;
      const double ur = (rd * rd) * ir2, ub = (bd * bd) * ib2;
      pc = R * iB;
      rl = TIER == 0 ? R * mean_Gh(ur) : (0.5 * R) * rcp_cheb(mean_F_wide(ur));
      ct = (TIER == 0 ? mean_F(ub) : mean_F_wide(ub)) * (iB * c0);
    } else {
      const double iB = 1.0 / B;
      rl = logavg_wide(P.r, Q.r);
      pc = R * iB;
      ct = 0.5 * c0 / logavg_wide(P.v[DIM], Q.v[DIM]);
    }
    double ua[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) ua[c] = P.v[c] + Q.v[c];
    const double fr = ua[0] * rl;
    f[0] = fr;
#pragma unroll
    for (int c = 0; c < DIM; ++c) f[1 + c] = (c == 0) ? fma(fr, ua[c], pc) : fr * ua[c];
    double uu = P.v[0] * Q.v[0];
#pragma unroll
    for (int c = 1; c < DIM; ++c) uu = fma(P.v[c], Q.v[c], uu);
    double ef = fma(2.0, uu, ct);
    if constexpr (S::EG) ef = fma(2.0, P.ph + Q.ph, ef);
    f[DIM + 1] = fma(fr, ef, pc * ua[0]);
    if constexpr (S::EG) x = (B * rl) * (P.ph - Q.ph);
  }
}

// The form (TIER) of a line's logarithmic means: how far apart its densities and B lie,
// from the high words (monotonic for positive values).  The polynomial forms are
// for positive numbers of ordinary size: their common reciprocal of (R B)^2 stays a
// normal number (FP32: so do the quotients).
template <int LAW, int DIM, int VK, int NQ>
__device__ __forceinline__ int line_form(const double* sq, const double* sx, int base, int sd) {
  int form = 0;
  if constexpr ((VK == VK_EC || VK == VK_EC32) && LAW != LAW_SW) {
    constexpr int npl = line_nodes(NQ, DIM);
    int rlo = 0x7fffffff, rhi = -0x7fffffff - 1, blo = rlo, bhi = rhi;
#pragma unroll
    for (int a = 0; a < NQ; ++a) {
      const int n = base + a * sd;
      const int hr = __double2hiint(sq[n]), hb = __double2hiint(sx[(VK == VK_EC ? DIM : 1) * npl + n]);
      rlo = min(rlo, hr);
      rhi = max(rhi, hr);
      blo = min(blo, hb);
      bhi = max(bhi, hb);
    }
    const double rmax = __hiloint2double(rhi + 1, 0), bmax = __hiloint2double(bhi + 1, 0);
    const double rmin = __hiloint2double(rlo, 0), bmin = __hiloint2double(blo, 0);
    constexpr int EX = VK == VK_EC32 ? 100 : 240;  // between 2^-EX and 2^EX
    const bool plain = min(rlo, blo) >= ((1023 - EX) << 20) && max(rhi, bhi) < ((1023 + EX) << 20);
    const bool near = plain && rmax < 1.2 * rmin && bmax < 1.2 * bmin;
    if constexpr (VK == VK_EC32)
      form = near ? 0 : 2;
    else
      form = near ? 0 : plain && rmax < 3.0 * rmin && bmax < 3.0 * bmin ? 1 : 2;
  }
  return form;
}

// every pair of the line, both nodes' rows of Cfd (in the parameters: constant-
// bank operands)
template <int LAW, int DIM, int VK, int NQ, int TIER>
__device__ __forceinline__ void line_pairs(const TendArgs& A, double c0, const double* sq, const double* sx, int base,
                                           int sd, const int* rot, int d, double (*T)[NSt<LAW, DIM>::v], double* X) {
  using S = LineShape<LAW, DIM, VK>;
  constexpr int NS = S::NS;
  constexpr int npl = line_nodes(NQ, DIM);
#pragma unroll
  for (int a = 0; a < NQ - 1; ++a) {
    LinePt<LAW, DIM, VK> P;
    line_load<LAW, DIM, VK, DIM == 3 && NQ >= 6>(P, sq, sx, npl, base + a * sd, rot, d);
#pragma unroll
    for (int b = a + 1; b < NQ; ++b) {
      LinePt<LAW, DIM, VK> Q;
      line_load<LAW, DIM, VK, DIM == 3 && NQ >= 6>(Q, sq, sx, npl, base + b * sd, rot, d);
      double f[NS], x = 0.0;
      line_pair<LAW, DIM, VK, TIER>(A.law, c0, d, P, Q, f, x);
      const double cab = A.cfd[a * NQ + b], cba = A.cfd[b * NQ + a];
      if constexpr (S::EG && (VK == VK_KG || VK == VK_KG32)) {
        // the fluctuation has no node factor: into the flux, as it cancels there
        const double fb = f[1] + x;
        f[1] = f[1] - x;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          T[a][s] = fma(cab, f[s], T[a][s]);
          T[b][s] = fma(cba, s == 1 ? fb : f[s], T[b][s]);
        }
      } else {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          T[a][s] = fma(cab, f[s], T[a][s]);
          T[b][s] = fma(cba, f[s], T[b][s]);
        }
        if constexpr (S::XTRA) {
          X[a] = fma(cab, x, X[a]);
          X[b] = fma(-cba, x, X[b]);
        }
      }
    }
  }
}

// Weak form: D^T-weighted flux rows of the line's nodes (Cw in the parameters),
// [m_n, m u_n + p n, (rho e + p) u_n] rotated
template <int DIM>
__device__ __forceinline__ void weak_row(const double* sq, const double* sx, int npl, int n, const int* rot, double* f) {
  f[0] = sq[(1 + rot[0]) * npl + n];
  const double un = __dmul_rn(f[0], sx[n]);
  f[1] = fma(f[0], un, sx[npl + n]);
#pragma unroll
  for (int c = 1; c < DIM; ++c) f[1 + c] = __dmul_rn(sq[(1 + rot[c]) * npl + n], un);
  f[DIM + 1] = __dmul_rn(sx[2 * npl + n], un);
}
template <int DIM, int NQ>
__device__ __forceinline__ void line_weak(const TendArgs& A, const double* sq, const double* sx, int base, int sd,
                                          const int* rot, double (*T)[DIM + 2]) {
  constexpr int npl = line_nodes(NQ, DIM);
#pragma unroll
  for (int m = 0; m < NQ; ++m) {
    double f[DIM + 2];
    weak_row<DIM>(sq, sx, npl, base + m * sd, rot, f);
#pragma unroll
    for (int a = 0; a < NQ; ++a)
#pragma unroll
      for (int s = 0; s < DIM + 2; ++s) T[a][s] = fma(A.cfd[a * NQ + m], f[s], T[a][s]);
  }
}

// ------------------------------------------------------------ face fluxes
// FP64 Rusanov flux of Euler, Euler-gravity and shallow water from rotated
// face states (src/numericalfluxes.jl:31-42).  Every product that an addition
// could absorb is either an explicit fma or an explicitly rounded product, so
// the result does not depend on what the compiler fuses where.
template <int LAW, int DIM>
__device__ __forceinline__ void line_rusanov(const LawP& L, double sgn, const double* qm, const double* am,
                                             const double* qp, const double* ap, double* nf) {
  const double rm = rcp_cheb(qm[0]), rp = rcp_cheb(qp[0]);
  double um[DIM], up[DIM], f[DIM + 2];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    um[c] = __dmul_rn(qm[1 + c], rm);
    up[c] = __dmul_rn(qp[1 + c], rp);
  }
  f[0] = qm[1] + qp[1];
  double wm, wp;
  if constexpr (LAW == LAW_SW) {
    const double hg = 0.5 * L.grav;
    f[1] = fma(__dmul_rn(hg, qm[0]), qm[0], __dmul_rn(__dmul_rn(hg, qp[0]), qp[0]));
    f[DIM + 1] = fma(um[0], qm[DIM + 1], __dmul_rn(up[0], qp[DIM + 1]));
    wm = sqrt_house(__dmul_rn(L.grav, qm[0]));
    wp = sqrt_house(__dmul_rn(L.grav, qp[0]));
  } else {
    const double g1 = L.gamma - 1.0;
    double tm = fma(-0.5, dot<DIM>(qm + 1, um), qm[DIM + 1]), tp = fma(-0.5, dot<DIM>(qp + 1, up), qp[DIM + 1]);
    if constexpr (LAW == LAW_EG) {
      tm = fma(-qm[0], am[0], tm);
      tp = fma(-qp[0], ap[0], tp);
    }
    const double pm = __dmul_rn(g1, tm), pp = __dmul_rn(g1, tp);
    f[1] = pm + pp;
    if (LAW == LAW_EG && L.pde) f[1] = f[1] - (am[DIM + 2] + ap[DIM + 2]);
    f[DIM + 1] = fma(um[0], qm[DIM + 1] + pm, __dmul_rn(up[0], qp[DIM + 1] + pp));
    wm = sqrt_house(__dmul_rn(__dmul_rn(L.gamma, pm), rm));
    wp = sqrt_house(__dmul_rn(__dmul_rn(L.gamma, pp), rp));
  }
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const double t = __dmul_rn(qp[1], up[c]);
    f[1 + c] = (c == 0) ? f[1] + fma(qm[1], um[0], t) : fma(qm[1], um[c], t);
  }
  const double hs = 0.5 * sgn, ws = -0.5 * dmax(fabs(um[0]) + wm, fabs(up[0]) + wp);
#pragma unroll
  for (int s = 0; s < DIM + 2; ++s) nf[s] = fma(ws, qp[s] - qm[s], __dmul_rn(hs, f[s]));
  if constexpr (LAW == LAW_SW) {
    // non-conservative surface term g h- (b+ - b-)/2 n (zero without bathymetry)
    nf[1] = fma(__dmul_rn(__dmul_rn(L.grav, qm[0]), hs), ap[0] - am[0], nf[1]);
  }
}

// Linear Euler-gravity: H = (rho e + p)_ref / rho_ref = Phi + g/(g-1) p_ref /
// rho_ref and the reference sound speed, from aux = [Phi, rho_ref, p_ref]
__device__ __forceinline__ double lin_enthalpy(double gg1, double Phi, double rho_ref, double p_ref, double* pr) {
  *pr = __dmul_rn(p_ref, rcp_cheb(rho_ref));
  return fma(gg1, *pr, Phi);
}

// boundarystate on rotated states: direction d, rot[c] the physical component
// of rotated component c, nc the rotated position of the normal component
template <int LAW, int DIM>
__device__ __forceinline__ void boundary_state_rot(const LawP& L, int d, const int* rot, int nc, double sgn, int tag,
                                                   const double* qm, double* qp) {
  constexpr int NS = NSt<LAW, DIM>::v;
#pragma unroll
  for (int s = 0; s < NS; ++s) qp[s] = qm[s];
  if (L.bc == BC_REFLECT) {
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      if (c == nc) qp[1 + c] = qm[1 + c] - 2.0 * (sgn * qm[1 + c]) * sgn;
  } else if (L.bc == BC_INFLOW_ZERO) {
    if (sgn * L.adv_u[d] <= 0.0) {
#pragma unroll
      for (int s = 0; s < NS; ++s) qp[s] = 0.0;
    }
  } else if (L.bc == BC_DIRICHLET) {
    const double* st = L.bc_state[tag == 1 ? 0 : 1];
    qp[0] = st[0];
    qp[DIM + 1] = st[DIM + 1];
#pragma unroll
    for (int c = 0; c < DIM; ++c) qp[1 + c] = st[1 + rot[c]];
  }
}

// The other numerical fluxes of a face node.  FP32-flux forms of Euler and
// Euler-gravity: components in x, y, z order with the direction a constant, so
// their FP32 sums round as in the node-per-thread kernels; else rotated
// (direction 0).
template <int LAW, int DIM, bool F32>
__device__ __forceinline__ void line_flux_dir(const LawP& L, int kind, int d, double sgn, const double* qm,
                                              const double* am, const double* qp, const double* ap, double* nf) {
  auto one = [&](auto dc) {
    constexpr int D_ = decltype(dc)::value;
    if (!F32 || !surface_flux32<LAW, DIM>(L, kind, D_, sgn, qm, am, qp, ap, nf))
      surface_flux<LAW, DIM>(L, kind, D_, sgn, qm, am, qp, ap, nf);
  };
  if constexpr (F32 && LAW != LAW_SW) {
    if (DIM > 2 && d == 2)
      one(std::integral_constant<int, (DIM > 2 ? 2 : 0)>{});
    else if (DIM > 1 && d == 1)
      one(std::integral_constant<int, (DIM > 1 ? 1 : 0)>{});
    else
      one(std::integral_constant<int, 0>{});
  } else {
    one(std::integral_constant<int, 0>{});
  }
}
// every flux, chosen at run time: one out-of-line copy
template <int LAW, int DIM, bool F32>
__device__ __noinline__ void line_flux_any(const LawP& L, int kind, int d, double sgn, const double* qm,
                                           const double* am, const double* qp, const double* ap, double* nf) {
  line_flux_dir<LAW, DIM, F32>(L, kind, d, sgn, qm, am, qp, ap, nf);
}
template <int LAW, int DIM, bool F32, int SF>
__device__ __forceinline__ void line_flux(const LawP& L, int kind, int d, double sgn, const double* qm,
                                          const double* am, const double* qp, const double* ap, double* nf) {
  if constexpr (SF >= 0)
    line_flux_dir<LAW, DIM, F32>(L, SF, d, sgn, qm, am, qp, ap, nf);
  else
    line_flux_any<LAW, DIM, F32>(L, kind, d, sgn, qm, am, qp, ap, nf);
}

// rotated component c of direction d: the normal component first
template <int DIM> __device__ __forceinline__ int line_rot(int c, int d) {
  const int r = c + d;
  return r >= DIM ? r - DIM : r;
}

// Per direction: line l's first node and node stride, in padded rows (P) or
// in the element's own node numbering
template <int NQ, int DIM>
__device__ __forceinline__ int line_base(int d, int l, int row) {
  if constexpr (DIM == 1) return 0;
  if constexpr (DIM == 2) return d == 0 ? row * l : l;
  return d == 0 ? row * l : d == 1 ? (l % NQ) + row * NQ * (l / NQ) : (l % NQ) + row * (l / NQ);
}
template <int NQ, int DIM>
__device__ __forceinline__ int line_stride(int d, int row) {
  return d == 0 ? 1 : d == 1 ? row : row * NQ;
}

template <int LAW, int DIM, int VK, int NQ, bool FUSE, int SF, bool PERSIST, bool SMALL = false>
__global__ void __launch_bounds__(SMALL ? small_threads(NQ, DIM) : fd_cfg(LAW, DIM, VK, NQ).max_threads,
                                  SMALL ? 1 : fd_cfg(LAW, DIM, VK, NQ).min_blocks)
    fd_kernel(const __grid_constant__ TendArgs A) {
  static_assert(!(SMALL && PERSIST), "one launch mode");
  using S = LineShape<LAW, DIM, VK>;
  constexpr int NS = S::NS;
  constexpr int NAM = NAuxMax<LAW, DIM>::v;
  constexpr int ROW = line_row(NQ);
  constexpr int NPL = line_nodes(NQ, DIM);
  constexpr int NP = ipow(NQ, DIM);
  constexpr int NFP = ipow(NQ, DIM - 1);
  constexpr int NXA = S::NXA;
  constexpr int DZ = DIM - 1;
  constexpr bool F32S = S::F32 && !S::SW;  // FP32 face sums: components in x, y, z order
  const int epi = A.epi;
  const int sflux = SF >= 0 ? SF : A.sflux;
  const int lin_sflux = SF >= 0 ? SF : A.lin_sflux;
  const int E = SMALL ? 1 : A.E;
  extern __shared__ double sm[];
  double* const sW = sm;  // Cw (the fused linear operator), lift
  constexpr int NB = fd_cfg(LAW, DIM, VK, NQ).bufs;
  static_assert(NB == 1 || NB == DIM, "one accumulator array, or one per direction");
  constexpr int slotsz = SMALL ? small_slot(NS, NXA, NQ, DIM, FUSE) : fd_slot(NS, NXA, NQ, DIM, NB, FUSE);
  const int tid = threadIdx.x, nth = blockDim.x;
  for (int t = tid; t < NQ * NQ + 1; t += nth) sW[t] = A.tab[NQ * NQ + t];
  double* const s0 = sm + NQ * NQ + 2;
  // SMALL: Cfd (Cw for the weak form), face fluxes, line forms, pair numbers, pair values
  constexpr int NLN = line_count(NQ, DIM), NPR = small_pairs(NQ);
  double* const sC = s0 + slotsz;
  double* const sF = sC + NQ * NQ;
  int* const sForm = (int*)(sF + 2 * NLN * NS);
  int* const sPair = sForm + NLN;
  double* const sV = sF + 2 * NLN * NS + (NLN + NPR + 1) / 2;
  if constexpr (SMALL) {
    for (int t = tid; t < NQ * NQ; t += nth) {
      sC[t] = A.tab[(VK == VK_WEAK ? NQ * NQ : 0) + t];
      const int a = t / NQ, b = t - a * NQ;
      if (a < b) sPair[a * NQ - a * (a + 1) / 2 + b - a - 1] = a * 16 + b;
    }
  }
  // regions of an element's slot
  constexpr int OX = NS * NPL;                       // point values, later the accumulators
  constexpr int OL = OX + NXA * NPL;                 // fused: linear p', H m_z
  constexpr int OT = OL + (FUSE ? 2 * NPL : 0);      // fused: the linear tendency (without its sources)
  constexpr int OB = OT + (FUSE ? NS * NPL : 0);     // the other directions' accumulators (NB > 1)
  const LawP& L = A.law;
  pdl_wait();
  auto tile_body = [&](const int tile) {
    const int ne = min(E, A.K - tile * E);  // elements of this tile
    const size_t g0 = (size_t)tile * E * NP;
    // rounds of the node loops: the CTA has a thread per line, so their count
    // is a constant and the loads of all rounds are issued before the first
    // is used
    constexpr int RN = SMALL ? 1 : (NQ + DIM - 1) / DIM;  // (SMALL: a thread per node)
    constexpr bool RUS = SF == F_RUSANOV && !S::F32;
    // ------------------------------------------------ this thread's line
    // lines ordered by direction, then element: the lanes of a warp mostly
    // share a direction, and the vertical lines (which carry the fused linear
    // operator) fill few warps
    const int nld = E * NFP;
    // (SMALL: the next NLN threads own the lines' second faces)
    const int side = SMALL && tid >= NLN;
    const int tl = side ? tid - NLN : tid;
    const int d = DIM == 3 ? (tl >= nld) + (tl >= 2 * nld) : (tl >= nld);
    const int es_ = (tl - d * nld) / NFP;
    const bool line = es_ < ne && tid < DIM * nld;
    const int es = line ? es_ : 0;  // a thread without a line works on the first element and stores nothing
    const int l = tl < DIM * nld ? tl - d * nld - es_ * NFP : 0;
    const int e = tile * E + es;
    const bool act = (A.dirs >> d) & 1;
    int rot[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) rot[c] = line_rot<DIM>(c, d);
    // its two faces: neighbours, then their traces (rotated; x, y, z order in
    // the FP32-flux forms).  A boundary face loads its own trace, so the loads
    // are free of branches.
    int nv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) nv[i] = __ldg(A.nbr + 6 * e + 2 * d + (SMALL && i == 0 ? side : i));
    const double gd = __ldg(A.ginv + 3 * e + d);
    double qp[2][NS], ap[2];
    size_t nid[2];
    auto face_load = [&](int i) {
      const bool inner = nv[i] > NBR_BOUNDARY + 64;
      const bool hi = inner != ((SMALL && i == 0 ? side : i) == 1);  // the trace lies at the element's last node of the line
      nid[i] = (size_t)(e + (inner ? nv[i] : 0)) * NP + line_base<NQ, DIM>(d, l, NQ) +
               (hi ? NQ - 1 : 0) * line_stride<NQ, DIM>(d, NQ);
      qp[i][0] = __ldg(A.q[0] + nid[i]);
#pragma unroll
      for (int c = 0; c < DIM; ++c) qp[i][1 + c] = __ldg(A.q[1 + (F32S ? c : rot[c])] + nid[i]);
      qp[i][DIM + 1] = __ldg(A.q[DIM + 1] + nid[i]);
      ap[i] = 0.0;
      if (LAW == LAW_EG || (S::SW && L.swtopo)) ap[i] = __ldg(A.aux + nid[i]);
    };
    // ------------------------------------------------------- point values
    {
      constexpr int NA = FUSE ? 3 : 1;  // Phi (bathymetry) [, rho_ref, p_ref]
      double q[RN][NS], al[RN][NA];
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const unsigned v = tid + r * nth;
        if (v < ne * NP) {
#pragma unroll
          for (int s = 0; s < NS; ++s) q[r][s] = __ldg(A.q[s] + g0 + v);
          al[r][0] = 0.0;
          if (LAW == LAW_EG || (S::SW && L.swtopo)) al[r][0] = __ldg(A.aux + g0 + v);
#pragma unroll
          for (int k = 1; k < NA; ++k) al[r][k] = __ldg(A.aux + (DIM + k) * A.stride + g0 + v);
        }
      }
      face_load(0);
      face_load(1);
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const unsigned v = tid + r * nth;
        if (v < ne * NP) {
          const unsigned en = v / NP, n = v - en * NP;
          const unsigned pn = n + (ROW - NQ) * (n / NQ);
          double* const sq = s0 + en * slotsz + pn;
          double* const sx = sq + OX;
          const double a0 = al[r][0];
#pragma unroll
          for (int s = 0; s < NS; ++s) sq[s * NPL] = q[r][s];
          float* const sf = (float*)(s0 + en * slotsz + OX + S::ND * NPL) + pn;
          if constexpr (S::SW) {
            if constexpr (S::F32) {
              const float hinv = 1.f / (float)q[r][0];
#pragma unroll
              for (int c = 0; c < DIM; ++c) sf[c * NPL] = (float)q[r][1 + c] * hinv;
              sf[DIM * NPL] = (float)q[r][DIM + 1] * hinv;
            } else {
              const double hh = 0.5 * rcp_cheb(q[r][0]);
#pragma unroll
              for (int c = 0; c < DIM + 1; ++c) sx[c * NPL] = q[r][1 + c] * hh;
            }
            sx[(S::ND - 1) * NPL] = a0;
          } else {
            const double rinv = rcp_cheb(q[r][0]);
            double u[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) u[c] = __dmul_rn(q[r][1 + c], rinv);
            double t = fma(-0.5, dot<DIM>(q[r] + 1, u), q[r][DIM + 1]);
            if constexpr (S::EG) t = fma(-q[r][0], a0, t);
            const double p = __dmul_rn(L.gamma - 1.0, t);
            if constexpr (S::F32) {
              sx[0] = p;
              if constexpr (VK == VK_EC32) {
                const double pr = __dmul_rn(p, rinv);
                sx[NPL] = 0.5 * rcp_cheb(pr);
                sx[2 * NPL] = pr;
              }
              if constexpr (S::EG) sx[(S::ND - 1) * NPL] = a0;
              const float rinvf = (float)rinv;
              float uu = 0.f;
#pragma unroll
              for (int c = 0; c < DIM; ++c) {
                const float uf = (float)q[r][1 + c] * rinvf;
                sf[c * NPL] = uf;
                uu += uf * uf;
              }
              sf[DIM * NPL] = (VK == VK_EC32) ? uu : (float)q[r][DIM + 1] * rinvf;
            } else if constexpr (VK == VK_WEAK) {
              sx[0] = rinv;
              sx[NPL] = L.pde ? p - __ldg(A.aux + (DIM + 2) * A.stride + g0 + v) : p;
              sx[2 * NPL] = q[r][DIM + 1] + p;
              sx[(S::ND - 1) * NPL] = 0.25 * a0;
            } else {
#pragma unroll
              for (int c = 0; c < DIM; ++c) sx[c * NPL] = 0.5 * u[c];
              if constexpr (VK == VK_KG) {
                sx[DIM * NPL] = 0.5 * p;
                sx[(DIM + 1) * NPL] = 0.5 * (q[r][DIM + 1] * rinv);
              } else {
                const double pr = __dmul_rn(p, rinv);
                sx[DIM * NPL] = rcp_cheb(pr);
                sx[(DIM + 1) * NPL] = pr;
              }
              if constexpr (S::EG) sx[(S::ND - 1) * NPL] = 0.25 * a0;
            }
          }
          if constexpr (FUSE) {
            // the linear operator's z flux row [m_z, 0, 0, p', H m_z]
            double pr;
            const double H = lin_enthalpy(A.lin_gg1, a0, al[r][1], al[r][2], &pr);
            sq[OL] = __dmul_rn(A.lin_law.gamma - 1.0, fma(-q[r][0], a0, q[r][DIM + 1]));
            sq[OL + NPL] = __dmul_rn(H, q[r][1 + DZ]);
          }
        }
      }
    }
    __syncthreads();
    // -------------------------------------------------- the line's tendency
    const double lift_end = sW[NQ * NQ];
    double* const sq = s0 + es * slotsz;
    double* const sx = sq + OX;
    const int base = line_base<NQ, DIM>(d, l, ROW), sd = line_stride<NQ, DIM>(d, ROW);
    constexpr bool XYZ = VK == VK_EC32 && !S::SW;  // accumulators in x, y, z order
    if constexpr (SMALL) {
      if (tid < NLN) sForm[tid] = line_form<LAW, DIM, VK, NQ>(sq, sx, base, sd);
      __syncthreads();
    }
    double T[NQ][NS], X[NQ];
#pragma unroll
    for (int a = 0; a < NQ; ++a) {
      X[a] = 0.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) T[a][s] = 0.0;
    }
    if (act) {
      // ---- the numerical fluxes at the line's ends, one lift_end * flux each (i: the
      // end; k: its place in the arrays above)
      auto own = [&](int i, double* qm, double* am) {
        const int nm = base + (i ? (NQ - 1) * sd : 0);
        qm[0] = sq[nm];
#pragma unroll
        for (int c = 0; c < DIM; ++c) qm[1 + c] = sq[(1 + (F32S ? c : rot[c])) * NPL + nm];
        qm[DIM + 1] = sq[(DIM + 1) * NPL + nm];
#pragma unroll
        for (int k = 0; k < NAM; ++k) am[k] = 0.0;
        if (LAW == LAW_EG || S::SW) {
          am[0] = sx[(S::ND - 1) * NPL + nm];
          if (LAW == LAW_EG && !S::F32) am[0] = 4.0 * am[0];
        }
      };
      auto bc = [&](int k, int i, const LawP& Lb, const double* qm, double* qb) {
        if constexpr (F32S) {
          const int id[3] = {0, 1, 2};
          boundary_state_rot<LAW, DIM>(Lb, d, id, d, i ? 1.0 : -1.0, nv[k] - NBR_BOUNDARY, qm, qb);
        } else {
          boundary_state_rot<LAW, DIM>(Lb, d, rot, 0, i ? 1.0 : -1.0, nv[k] - NBR_BOUNDARY, qm, qb);
        }
      };
      // pde_level_balance: the reference state too
      auto aux = [&](int f, int i, double* am, double* apv) {
#pragma unroll
        for (int k = 0; k < NAM; ++k) apv[k] = 0.0;
        apv[0] = ap[f];
        if (LAW == LAW_EG && (RUS ? L.pde != 0 : A.naux_nl > 1)) {
          const size_t mid = (size_t)e * NP + line_base<NQ, DIM>(d, l, NQ) +
                             (size_t)(i ? (NQ - 1) : 0) * line_stride<NQ, DIM>(d, NQ);
#pragma unroll
          for (int k = 1; k < NAM; ++k)
            if (k < A.naux_nl) {
              am[k] = __ldg(A.aux + k * A.stride + mid);
              apv[k] = __ldg(A.aux + k * A.stride + nid[f]);
            }
        }
      };
      if constexpr (SMALL) {
        if (tid < 2 * NLN) {
          const double sgn = side ? 1.0 : -1.0;
          double qm[NS], am[NAM], apv[NAM], nf[NS];
          own(side, qm, am);
          if (nv[0] <= NBR_BOUNDARY + 64) bc(0, side, L, qm, qp[0]);
          aux(0, side, am, apv);
          if constexpr (RUS)
            line_rusanov<LAW, DIM>(L, sgn, qm, am, qp[0], apv, nf);
          else
            line_flux<LAW, DIM, S::F32, SF>(L, sflux, d, sgn, qm, am, qp[0], apv, nf);
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            double f = nf[s];
            if constexpr (F32S && !XYZ) {  // fluxes in x, y, z order, sums rotated
              if (s > 0 && s <= DIM) {
                f = nf[1];
#pragma unroll
                for (int k = 1; k < DIM; ++k)
                  if (rot[s - 1] == k) f = nf[1 + k];
              }
            }
            sF[s * 2 * NLN + tid] = __dmul_rn(-lift_end, f);
          }
        }
      } else {
        double qm[2][NS], am[2][NAM], apv[2][NAM], nf[2][NS];
        // both ends in one stretch of code: their chains overlap
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          own(i, qm[i], am[i]);
          if (nv[i] <= NBR_BOUNDARY + 64) bc(i, i, L, qm[i], qp[i]);
          aux(i, i, am[i], apv[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const double sgn = i ? 1.0 : -1.0;
          if constexpr (RUS)
            line_rusanov<LAW, DIM>(L, sgn, qm[i], am[i], qp[i], apv[i], nf[i]);
          else
            line_flux<LAW, DIM, S::F32, SF>(L, sflux, d, sgn, qm[i], am[i], qp[i], apv[i], nf[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          double(&Te)[NS] = T[i ? NQ - 1 : 0];
#pragma unroll
          for (int s = 0; s < NS; ++s) Te[s] = __dmul_rn(-lift_end, nf[i][s]);
          if constexpr (F32S && !XYZ) {  // fluxes in x, y, z order, accumulators rotated
#pragma unroll
            for (int c = 0; c < DIM; ++c) {
              double f = nf[i][1];
#pragma unroll
              for (int k = 1; k < DIM; ++k)
                if (rot[c] == k) f = nf[i][1 + k];
              Te[1 + c] = __dmul_rn(-lift_end, f);
            }
          }
        }
      }
    }
    if constexpr (FUSE) {
      // ---- the weak-form linear operator along the vertical lines: D^T of
      // the staged flux rows, the faces from the traces above
      if (d == DZ && line) {
        const double g1 = A.lin_law.gamma - 1.0;
        double fz[NQ][3];
#pragma unroll
        for (int a = 0; a < NQ; ++a) {
          const int n = base + a * sd;
          fz[a][0] = sq[(1 + DZ) * NPL + n];
          fz[a][1] = sq[OL + n];
          fz[a][2] = sq[OL + NPL + n];
        }
        double W[2][NS];  // lift_end * numerical flux at the ends, rotated
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int nm = base + (i ? (NQ - 1) * sd : 0);
          const double sgn = i ? 1.0 : -1.0;
          const bool inner = nv[i] > NBR_BOUNDARY + 64;
          const size_t mid = (size_t)e * NP + l + (i ? (NQ - 1) * NFP : 0);
          double qo[NS], qn[NS], Pn = inner ? ap[i] : __ldg(A.aux + mid);
          qo[0] = sq[nm];
#pragma unroll
          for (int c = 0; c < DIM; ++c) qo[1 + c] = sq[(1 + rot[c]) * NPL + nm];
          qo[DIM + 1] = sq[(DIM + 1) * NPL + nm];
          if (inner) {
            // (the traces above are in x, y, z order in the FP32-flux forms)
#pragma unroll
            for (int s = 0; s < NS; ++s) qn[s] = qp[i][s];
            if constexpr (F32S) {
              qn[1] = qp[i][1 + DZ];
#pragma unroll
              for (int c = 1; c < DIM; ++c) qn[1 + c] = qp[i][c];
            }
          } else {
            boundary_state_rot<LAW_LEG, DIM>(A.lin_law, d, rot, 0, sgn, nv[i] - NBR_BOUNDARY, qo, qn);
          }
          const double rm = __ldg(A.aux + (1 + DIM) * A.stride + mid), pm = __ldg(A.aux + (2 + DIM) * A.stride + mid);
          const size_t nn = inner ? nid[i] : mid;
          const double rp = __ldg(A.aux + (1 + DIM) * A.stride + nn), pp = __ldg(A.aux + (2 + DIM) * A.stride + nn);
          double nf[NS];
          if constexpr (SF == F_RUSANOV) {
            double prm, prp;
            lin_enthalpy(A.lin_gg1, 0.0, rm, pm, &prm);
            const double Hp = lin_enthalpy(A.lin_gg1, Pn, rp, pp, &prp);
            const double pl = __dmul_rn(g1, fma(-qn[0], Pn, qn[DIM + 1]));
            const double hs = 0.5 * sgn;
            // max(sqrt a, sqrt b) = sqrt(max(a, b))
            const double ws = -0.5 * sqrt_house(__dmul_rn(A.lin_law.gamma, dmax(prm, prp)));
#pragma unroll
            for (int s = 0; s < NS; ++s) nf[s] = __dmul_rn(ws, qn[s] - qo[s]);
            nf[0] = fma(hs, qo[1] + qn[1], nf[0]);
            nf[1] = fma(hs, fz[i ? NQ - 1 : 0][1] + pl, nf[1]);
            nf[DIM + 1] = fma(hs, fma(Hp, qn[1], fz[i ? NQ - 1 : 0][2]), nf[DIM + 1]);
          } else {
            double bm[6], bp[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) bm[k] = bp[k] = 0.0;
            bm[0] = __ldg(A.aux + mid);
            bm[1 + DIM] = rm;
            bm[2 + DIM] = pm;
            bp[0] = Pn;
            bp[1 + DIM] = rp;
            bp[2 + DIM] = pp;
            surface_flux<LAW_LEG, DIM>(A.lin_law, lin_sflux, 0, sgn, qo, bm, qn, bp, nf);
          }
#pragma unroll
          for (int s = 0; s < NS; ++s) W[i][s] = __dmul_rn(lift_end, nf[s]);
        }
#pragma unroll
        for (int a = 0; a < NQ; ++a) {
          double t[NS];  // rotated: [rho, m_z, m_x, m_y, rho e]
#pragma unroll
          for (int s = 0; s < NS; ++s) t[s] = a == 0 ? -W[0][s] : a == NQ - 1 ? -W[1][s] : 0.0;
#pragma unroll
          for (int m = 0; m < NQ; ++m) {
            const double c = sW[a * NQ + m];
            t[0] = fma(c, fz[m][0], t[0]);
            t[1] = fma(c, fz[m][1], t[1]);
            t[DIM + 1] = fma(c, fz[m][2], t[DIM + 1]);
          }
          double* const o = sq + OT + base + a * sd;
          o[0] = __dmul_rn(gd, t[0]);
          o[(1 + DZ) * NPL] = __dmul_rn(gd, t[1]);
#pragma unroll
          for (int c = 1; c < DIM; ++c) o[c * NPL] = __dmul_rn(gd, t[1 + c]);
          o[(DIM + 1) * NPL] = __dmul_rn(gd, t[DIM + 1]);
        }
      }
    }
    int form = 0;
    if constexpr (!SMALL) form = line_form<LAW, DIM, VK, NQ>(sq, sx, base, sd);
    // FP32 flux: a warp with a line of form 2 takes it for all of them, not one form
    // after the other (3-D N = 6, 8x6x4 elements: 115 -> 109 us per ARK23 step); a near
    // line's pairs come out the same to the bit (tests/test_fp32flux_lines.py)
    if constexpr (!SMALL && VK == VK_EC32 && !S::SW) form = __any_sync(0xffffffffu, form) ? 2 : 0;
    double Ts[NS];  // SMALL: the node's sums
    if constexpr (SMALL) {
      const int n0 = tid < NP ? tid : 0, i0 = n0 % NQ, i1 = n0 / NQ % NQ, i2 = n0 / (NQ * NQ);
      const int pn = n0 + (ROW - NQ) * (n0 / NQ);
      constexpr int DB = VK == VK_WEAK ? DIM : small_batch(NQ, DIM), NT = DB * NFP * NPR;
      const double c0 = (VK == VK_EC && !S::SW) ? 2.0 / (L.gamma - 1.0) : S::SW ? 0.5 * L.grav : 1.0 / (L.gamma - 1.0);
#pragma unroll
      for (int d0 = 0; d0 < DIM; d0 += DB) {
        if constexpr (VK != VK_WEAK) {
          if (d0 > 0) __syncthreads();
#pragma unroll 1
          for (int t = tid; t < NT; t += nth) {
            const int td = t / (NFP * NPR), r = t - td * (NFP * NPR), pi = r / NFP, tln = r - pi * NFP, dd = d0 + td;
            if (!((A.dirs >> dd) & 1)) continue;
            int rt[DIM];
#pragma unroll
            for (int c = 0; c < DIM; ++c) rt[c] = line_rot<DIM>(c, dd);
            const int b0 = line_base<NQ, DIM>(dd, tln, ROW), st = line_stride<NQ, DIM>(dd, ROW), ab = sPair[pi];
            LinePt<LAW, DIM, VK> P, Q;
            line_load<LAW, DIM, VK, false>(P, sq, sx, NPL, b0 + (ab >> 4) * st, rt, dd);
            line_load<LAW, DIM, VK, false>(Q, sq, sx, NPL, b0 + (ab & 15) * st, rt, dd);
            double f[NS], x = 0.0;
            if constexpr (VK == VK_EC && !S::SW) {
              const int fo = sForm[dd * NFP + tln];
              if (fo == 0)
                line_pair<LAW, DIM, VK, 0>(L, c0, dd, P, Q, f, x);
              else if (fo == 1)
                line_pair<LAW, DIM, VK, 1>(L, c0, dd, P, Q, f, x);
              else
                line_pair<LAW, DIM, VK, 2>(L, c0, dd, P, Q, f, x);
            } else if constexpr (VK == VK_EC32 && !S::SW) {
              if (sForm[dd * NFP + tln] == 0)
                line_pair<LAW, DIM, VK, 0>(L, c0, dd, P, Q, f, x);
              else
                line_pair<LAW, DIM, VK, 2>(L, c0, dd, P, Q, f, x);
            } else {
              line_pair<LAW, DIM, VK, 0>(L, c0, dd, P, Q, f, x);
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) sV[s * NT + t] = f[s];
            if constexpr (S::XTRA) sV[NS * NT + t] = x;
          }
        }
        __syncthreads();
#pragma unroll
        for (int dd = d0; dd < d0 + DB && dd < DIM; ++dd) {
          double t[NS];
#pragma unroll
          for (int s = 0; s < NS; ++s) t[s] = 0.0;
          if (tid < NP && ((A.dirs >> dd) & 1)) {
            const int a = dd == 0 ? i0 : dd == 1 ? i1 : i2;
            const int ln = DIM == 2 ? (dd == 0 ? i1 : i0) : dd == 0 ? i1 + NQ * i2 : dd == 1 ? i0 + NQ * i2 : i0 + NQ * i1;
            if (a == 0 || a == NQ - 1) {
              const int fc = (a == 0 ? 0 : NLN) + dd * NFP + ln;
#pragma unroll
              for (int s = 0; s < NS; ++s) t[s] = sF[s * 2 * NLN + fc];
            }
            if constexpr (VK == VK_WEAK) {
              int rt[DIM];
#pragma unroll
              for (int c = 0; c < DIM; ++c) rt[c] = line_rot<DIM>(c, dd);
              const int b0 = line_base<NQ, DIM>(dd, ln, ROW), st = line_stride<NQ, DIM>(dd, ROW);
#pragma unroll
              for (int m = 0; m < NQ; ++m) {
                double f[NS];
                weak_row<DIM>(sq, sx, NPL, b0 + m * st, rt, f);
                const double c = sC[a * NQ + m];
#pragma unroll
                for (int s = 0; s < NS; ++s) t[s] = fma(c, f[s], t[s]);
              }
            } else {
              double X = 0.0;
#pragma unroll
              for (int b = 0; b < NQ; ++b) {
                if (b == a) continue;
                const int lo = b < a ? b : a, hi = b < a ? a : b;
                const double* const v = sV + ((dd - d0) * NPR + lo * NQ - lo * (lo + 1) / 2 + hi - lo - 1) * NFP + ln;
                const double c = sC[a * NQ + b];
                double f[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) f[s] = v[s * NT];
                if constexpr (S::EG && (VK == VK_KG || VK == VK_KG32)) {
                  const double x = v[NS * NT];
                  f[1] = b < a ? f[1] + x : f[1] - x;
                } else if constexpr (S::XTRA) {
                  X = fma(b < a ? -c : c, v[NS * NT], X);
                }
#pragma unroll
                for (int s = 0; s < NS; ++s) t[s] = fma(c, f[s], t[s]);
              }
              if constexpr (S::XTRA && VK != VK_KG && VK != VK_KG32) {
                if constexpr (S::SW)
                  X = L.swtopo ? __dmul_rn(X, 0.5 * L.grav * sq[pn]) : 0.0;
                else if constexpr (VK == VK_EC)
                  X = __dmul_rn(X, sx[(DIM + 1) * NPL + pn]);
                else if constexpr (VK == VK_EC32)
                  X = __dmul_rn(X, sx[2 * NPL + pn]);
                t[XYZ ? 1 + dd : 1] -= X;
              }
            }
            const double gn = __ldg(A.ginv + 3 * e + dd);
#pragma unroll
            for (int s = 0; s < NS; ++s) t[s] = __dmul_rn(t[s], gn);
          }
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const int c = (s == 0 || s == DIM + 1 || XYZ) ? s : 1 + (s - 1 + dd) % DIM;
            Ts[c] = dd == 0 ? t[s] : Ts[c] + t[s];
          }
        }
      }
    } else if (act) {
      // ---- two-point fluxes of the line's pairs, or the weak form's rows
      if constexpr (VK == VK_WEAK) {
        line_weak<DIM, NQ>(A, sq, sx, base, sd, rot, T);
      } else if constexpr (VK == VK_EC && !S::SW) {
        const double c0 = 2.0 / (L.gamma - 1.0);
        if (form == 0)
          line_pairs<LAW, DIM, VK, NQ, 0>(A, c0, sq, sx, base, sd, rot, d, T, X);
        else if (form == 1)
          line_pairs<LAW, DIM, VK, NQ, 1>(A, c0, sq, sx, base, sd, rot, d, T, X);
        else
          line_pairs<LAW, DIM, VK, NQ, 2>(A, c0, sq, sx, base, sd, rot, d, T, X);
      } else if constexpr (VK == VK_EC32 && !S::SW) {
        const double c0 = 1.0 / (L.gamma - 1.0);
        if (form == 0)
          line_pairs<LAW, DIM, VK, NQ, 0>(A, c0, sq, sx, base, sd, rot, d, T, X);
        else
          line_pairs<LAW, DIM, VK, NQ, 2>(A, c0, sq, sx, base, sd, rot, d, T, X);
      } else {
        const double c0 = S::SW ? 0.5 * L.grav : 1.0 / (L.gamma - 1.0);
        line_pairs<LAW, DIM, VK, NQ, 0>(A, c0, sq, sx, base, sd, rot, d, T, X);
      }
#pragma unroll
      for (int a = 0; a < NQ; ++a) {
        if constexpr (S::XTRA && VK != VK_KG && VK != VK_KG32) {
          const int n = base + a * sd;
          double t = X[a];
          if constexpr (S::SW)
            t = L.swtopo ? __dmul_rn(t, 0.5 * L.grav * sq[n]) : 0.0;
          else if constexpr (VK == VK_EC)
            t = __dmul_rn(t, sx[(DIM + 1) * NPL + n]);
          else if constexpr (VK == VK_EC32)
            t = __dmul_rn(t, sx[2 * NPL + n]);
          if constexpr (XYZ) {
#pragma unroll
            for (int c = 0; c < DIM; ++c)
              if (c == d) T[a][1 + c] -= t;
          } else {
            T[a][1] -= t;
          }
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) T[a][s] = __dmul_rn(T[a][s], gd);
      }
    }
    if constexpr (!SMALL) __syncthreads();  // the point values are dead: their region takes the sums
    if constexpr (SMALL) {
    } else if constexpr (NB > 1) {
      if (line) {  // (an inactive direction writes its zeros)
        double* const B = d == 0 ? sx : sq + OB + (d - 1) * NS * NPL;
#pragma unroll
        for (int a = 0; a < NQ; ++a)
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const int c = (s == 0 || s == DIM + 1 || XYZ) ? s : 1 + rot[s - 1];
            B[c * NPL + base + a * sd] = T[a][s];
          }
      }
    } else {
#pragma unroll
      for (int dd = 0; dd < DIM; ++dd) {
        if (dd > 0) __syncthreads();
        if (line && d == dd) {
#pragma unroll
          for (int a = 0; a < NQ; ++a)
#pragma unroll
            for (int s = 0; s < NS; ++s) {
              const int c = (s == 0 || s == DIM + 1 || XYZ) ? s : 1 + (s - 1 + dd) % DIM;
              double* const o = sx + c * NPL + base + a * sd;
              *o = dd == 0 ? T[a][s] : *o + T[a][s];
            }
        }
      }
    }
    // the epilogue's inputs, loaded before the barrier; fused: grad Phi too
    constexpr int NIN = FUSE ? 2 : 1;
    double in[RN][NIN][NS], gp[RN][DIM];
    {
      if constexpr (VK == VK_WEAK) {
#pragma unroll
        for (int r = 0; r < RN; ++r) {
          const unsigned v = tid + r * nth;
          if (v < ne * NP) {
#pragma unroll
            for (int k = 0; k < DIM; ++k) gp[r][k] = __ldg(A.aux + (1 + k) * A.stride + g0 + v);
          }
        }
      }
      const bool rd = FUSE || epi == EPI_ADD || (epi == EPI_LSRK && A.a != 0.0) || epi == EPI_SUBOUT2 || epi == EPI_RLSRK;
      const bool o2 = epi == EPI_SUBOUT2 || epi == EPI_RLSRK;
      if (rd) {
#pragma unroll
        for (int r = 0; r < RN; ++r) {
          const unsigned v = tid + r * nth;
          if (v < ne * NP) {
            if constexpr (FUSE) {
#pragma unroll
              for (int k = 0; k < DIM; ++k) gp[r][k] = __ldg(A.aux + (1 + k) * A.stride + g0 + v);
            }
#pragma unroll
            for (int i = 0; i < NIN; ++i)
              if (!FUSE || A.accin[i][0]) {
#pragma unroll
                for (int s = 0; s < NS; ++s)
                  in[r][i][s] = (FUSE ? A.accin[i][s] : o2 ? A.out2[s] : A.out[s])[g0 + v];
              }
          }
        }
      }
    }
    if constexpr (!SMALL) __syncthreads();
    // ----------------------------------------------------------- epilogue
    const bool cor = L.src == SRC_CORIOLIS && ((A.dirs >> DZ) & 1);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const unsigned v = tid + r * nth;
      if (v >= ne * NP) break;
      const unsigned en = v / NP, n = v - en * NP;
      const double* const qn = s0 + en * slotsz + n + (ROW - NQ) * (n / NQ);  // qn[s * NPL]: own state
      const size_t gid = g0 + v;
      double T[NS], TL[NS];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        if constexpr (SMALL) {
          T[s] = Ts[s];
          continue;
        }
        T[s] = qn[OX + s * NPL];
        if constexpr (NB > 1) {
#pragma unroll
          for (int k = 1; k < DIM; ++k) T[s] += qn[OB + ((k - 1) * NS + s) * NPL];
        }
      }
      auto coriolis = [&](const double* om, double* t) {
        if constexpr (DIM == 3) {
          const double m0 = qn[NPL], m1 = qn[2 * NPL], m2 = qn[3 * NPL];
          t[1] -= fma(om[1], m2, -__dmul_rn(om[2], m1));
          t[2] -= fma(om[2], m0, -__dmul_rn(om[0], m2));
          t[3] -= fma(om[0], m1, -__dmul_rn(om[1], m0));
        } else {
          t[1] = fma(om[2], qn[2 * NPL], t[1]);
          t[2] = fma(-om[2], qn[NPL], t[2]);
        }
      };
      if (cor) coriolis(L.omega, T);
      if constexpr (VK == VK_WEAK) {  // -rho grad Phi (the pair fluxes carry it otherwise)
        if ((A.dirs >> DZ) & 1) {
          const double rho = L.pde ? qn[0] - __ldg(A.aux + (DIM + 1) * A.stride + gid) : qn[0];
#pragma unroll
          for (int k = 0; k < DIM; ++k) T[1 + k] = fma(-rho, gp[r][k], T[1 + k]);
        }
      }
      if constexpr (FUSE) {
#pragma unroll
        for (int s = 0; s < NS; ++s) TL[s] = qn[OT + s * NPL];
#pragma unroll
        for (int k = 0; k < DIM; ++k) TL[1 + k] = fma(-qn[0], gp[r][k], TL[1 + k]);
        if (A.lin_law.src == SRC_CORIOLIS) coriolis(A.lin_law.omega, TL);
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (A.acc[j][0]) {
            const bool rd = A.accin[j][0] != nullptr;  // accumulators read and written come first (run_fused)
#pragma unroll
            for (int s = 0; s < NS; ++s) {
              const double b = rd ? in[r][j < NIN ? j : NIN - 1][s] : qn[s * NPL];
              A.acc[j][s][gid] = fma(A.adt, fma(A.ca[j], T[s] - TL[s], __dmul_rn(A.cb[j], TL[s])), b);
            }
          }
      } else if (epi == EPI_LSRK) {
        const double bdt = A.dte ? A.bdt * A.dte[tile * E + en] : A.bdt;
        // first stage (a = 0): the previous increment is not read, so stale or
        // never-written storage cannot leak into the step
        if (A.a != 0.0) {
#pragma unroll
          for (int s = 0; s < NS; ++s) T[s] = fma(A.a, in[r][0][s], T[s]);
        }
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          A.out[s][gid] = T[s];
          A.out2[s][gid] = fma(bdt, T[s], qn[s * NPL]);
        }
      } else if (epi == EPI_SET) {
#pragma unroll
        for (int s = 0; s < NS; ++s) A.out[s][gid] = T[s];
      } else if (epi == EPI_ADD) {
#pragma unroll
        for (int s = 0; s < NS; ++s) A.out[s][gid] = in[r][0][s] + T[s];
      } else if (epi == EPI_SUBOUT2) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          A.out[s][gid] = T[s];
          A.out2[s][gid] = in[r][0][s] - T[s];
        }
      } else if (epi == EPI_RLSRK) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          A.out[s][gid] = T[s];
          A.out2[s][gid] = fma(A.a, in[r][0][s], T[s]);
        }
      } else {  // EPI_ARK after a separate explicit launch: out holds N(Q), T = L(Q)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (A.acc[j][0]) {
#pragma unroll
            for (int s = 0; s < NS; ++s) {
              const double b = A.accin[j][0] ? A.accin[j][s][gid] : qn[s * NPL];
              A.acc[j][s][gid] = b + A.adt * (A.ca[j] * (A.out[s][gid] - T[s]) + A.cb[j] * T[s]);
            }
          }
      }
    }
  };
  if constexpr (PERSIST) {
    const int ntiles = (A.K + E - 1) / E;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      tile_body(tile);
      __syncthreads();  // the next tile restages shared memory
    }
  } else {
    tile_body(blockIdx.x);
  }
  pdl_trigger();
}

template <int LAW, int DIM, int VK, int NQ, bool FUSE = false, int SF = -1, bool PERSIST = false>
void fd_launch(const TendArgs& A, int grid, int block, size_t smem, cudaStream_t st) {
  if constexpr (!PERSIST && fd_has_small(LAW, DIM, VK, SF)) {
    if (A.small) {
      using S = LineShape<LAW, DIM, VK>;
      constexpr size_t bytes =
          sizeof(double) * small_doubles(S::NS, S::NXA, NQ, DIM, FUSE, VK != VK_WEAK);
      static SmemLimit small_limit;
      raise_smem(fd_kernel<LAW, DIM, VK, NQ, FUSE, SF, false, true>, small_limit, bytes);
      launch_maybe_pdl(fd_kernel<LAW, DIM, VK, NQ, FUSE, SF, false, true>, dim3(A.K), dim3(A.small), bytes, st, A);
      return;
    }
  }
  static SmemLimit limit;
  raise_smem(fd_kernel<LAW, DIM, VK, NQ, FUSE, SF, PERSIST>, limit, smem);
  launch_maybe_pdl(fd_kernel<LAW, DIM, VK, NQ, FUSE, SF, PERSIST>, dim3(grid), dim3(block), smem, st, A);
}

// the kernel of a node count (persistent ones: Nq = 4..6)
template <int LAW, int DIM, int VK, bool FUSE, int SF, bool PERSIST> tend_launch_fn fd_pick(int nq) {
  if constexpr (!PERSIST) {
    if (nq == 2) return fd_launch<LAW, DIM, VK, 2, FUSE, SF>;
    if (nq == 3) return fd_launch<LAW, DIM, VK, 3, FUSE, SF>;
    if (nq == 7) return fd_launch<LAW, DIM, VK, 7, FUSE, SF>;
    if (nq == 8) return fd_launch<LAW, DIM, VK, 8, FUSE, SF>;
  }
  if (nq == 4) return fd_launch<LAW, DIM, VK, 4, FUSE, SF, PERSIST>;
  if (nq == 5) return fd_launch<LAW, DIM, VK, 5, FUSE, SF, PERSIST>;
  if (nq == 6) return fd_launch<LAW, DIM, VK, 6, FUSE, SF, PERSIST>;
  return nullptr;
}

tend_launch_fn pick_fd(int law, int dim, int vk, int nq, int sflux);
tend_launch_fn pick_fd_fused(int dim, int vk, int nq, int sflux, int lin_sflux);
tend_launch_fn pick_fd_persistent(int law, int dim, int vk, int nq, int sflux, bool fused, int lin_sflux);

}  // namespace atb
