// ---------------------------------------------------------------------------
// Flux core of the FP64 step: the record accesses and the per-face arithmetic
// that the face kernels (kernels.cu) and the march kernel (march.cu, with its
// tiles' branch bits in tiles.cu) share. Every sum and product that a compiler
// could contract in one kernel and not in another is written as an explicit
// rounding (fma, __dmul_rn, __dadd_rn), so that all of them compute a face's flux
// bit for bit alike.
// ---------------------------------------------------------------------------
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

struct __align__(32) d4 {
  double x, y, z, w;
};

// Records of four doubles move as one 256-bit access (a whole 32-byte
// sector per thread; every record array is 32-byte aligned): half the load
// and store instructions of two 128-bit halves (step 0.541 -> 0.502 ms).
// Read-only data: non-coherent load the compiler may schedule freely.
__device__ __forceinline__ d4 ld4(const void* base, long long i) {
  const double* p = reinterpret_cast<const double*>(base) + 4 * i;
  d4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
      : "l"(p));
  return v;
}
// Coherent load, for data the same kernel also writes (kept in order).
__device__ __forceinline__ d4 ld4rw(const void* base, long long i) {
  const double* p = reinterpret_cast<const double*>(base) + 4 * i;
  d4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st4(void* base, long long i, const d4& v) {
  double* p = reinterpret_cast<double*>(base) + 4 * i;
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z),
               "d"(v.w)
               : "memory");
}

// The same pointer, opaque to the compiler, so that a load through it is not
// merged with an earlier load of the same address (a deliberate re-read).
template <typename T>
__device__ __forceinline__ const T* launder(const T* p) {
  asm("mov.b64 %0, %0;" : "+l"(p));
  return p;
}

// Ghost state from its owner. FL = 0 (GPU kernels, update_unstructured_bcs
// in LBFS.cu:1228-1301): bc1 holds the Dirichlet target, the raw value or for
// the parabolic inlet (vel type 9) the profile 16 u (H/2+y)(H/2-y)(H/2+z)(H/2-z)/H^4
// in x. FL = 1 (CPU Solver, Solution::update_unstructured_bcs,
// Solution.cpp:759-833): rho 1 mirror, 2 copy, 6 and 7 the value; velocity 1
// mirror, 2 copy, 6 the value, 8 (u, -v, w) of the owner.
template <int FL>
__device__ __forceinline__ d4 ghost_state(const d4& q, const d4& tgt, int types) {
  const int rt = types & 0xff, vt = types >> 8;
  d4 g;
  if (FL == 1) {
    g.w = rt == 1 ? tgt.w - (q.w - tgt.w) : (rt == 2 ? q.w : tgt.w);
    if (vt == 1) {
      g.x = tgt.x - (q.x - tgt.x);
      g.y = tgt.y - (q.y - tgt.y);
      g.z = tgt.z - (q.z - tgt.z);
    } else if (vt == 2) {
      g.x = q.x;
      g.y = q.y;
      g.z = q.z;
    } else if (vt == 8) {
      g.x = q.x;
      g.y = -q.y;
      g.z = q.z;
    } else {
      g.x = tgt.x;
      g.y = tgt.y;
      g.z = tgt.z;
    }
    return g;
  }
  g.w = (rt == 1) ? tgt.w - (q.w - tgt.w) : q.w;
  if (vt == 2) {
    g.x = q.x;
    g.y = q.y;
    g.z = q.z;
  } else {
    g.x = tgt.x - (q.x - tgt.x);
    g.y = tgt.y - (q.y - tgt.y);
    g.z = tgt.z - (q.z - tgt.z);
  }
  return g;
}

// Gradients as 12 doubles: rho, u, v, w, each (x, y, z).
__device__ __forceinline__ void load_grad(const void* base, int c, double g[12]) {
  const d4 a0 = ld4(base, 3LL * c), a1 = ld4(base, 3LL * c + 1), a2 = ld4(base, 3LL * c + 2);
  g[0] = a0.x; g[1] = a0.y; g[2] = a0.z; g[3] = a0.w;
  g[4] = a1.x; g[5] = a1.y; g[6] = a1.z; g[7] = a1.w;
  g[8] = a2.x; g[9] = a2.y; g[10] = a2.z; g[11] = a2.w;
}

// Ghost gradient. FL = 0 (get_bc_gradients, LBFS.cu:1306-1416): Dirichlet
// 2 (bc - q_owner) / |d| * d_hat from the raw boundary value (bc2 = (d_hat,
// |d|)); Neumann the owner's gradient times (1 - |n|) componentwise (bc3).
// FL = 1 (gradients::Get_LS_Gradients and get_ghost_grads,
// gradients.cpp:395-506,592-648): Dirichlet (rho 1, velocity 1 and 8) along
// the face normal (bc2 = (n, |d|)), Neumann times (1 - n) (bc3), types 6 zero,
// rho 7 the owner's gradient.
template <int FL>
__device__ __forceinline__ void ghost_grad(const d4& q, const double go[12], const d4& bv,
                                           const d4& dd, const d4& nm, int types,
                                           double g[12]) {
  const int rt = types & 0xff, vt = types >> 8;
  const double dir[3] = {dd.x, dd.y, dd.z}, m[3] = {nm.x, nm.y, nm.z};
  const double dq[4] = {2 * (bv.w - q.w), 2 * (bv.x - q.x), 2 * (bv.y - q.y), 2 * (bv.z - q.z)};
  if constexpr (FL == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const int t = f == 0 ? rt : vt;
#pragma unroll
      for (int c = 0; c < 3; c++)
        g[3 * f + c] = (t == 1 || (f > 0 && t == 8)) ? dq[f] / dd.w * dir[c]
                       : t == 2                      ? go[3 * f + c] * m[c]
                       : t == 7                      ? go[3 * f + c]
                                                     : 0.0;
    }
  } else {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const bool dirichlet = (f == 0) ? (rt == 1) : (vt != 2);
#pragma unroll
      for (int c = 0; c < 3; c++)
        g[3 * f + c] = dirichlet ? dq[f] / dd.w * dir[c] : go[3 * f + c] * m[c];
    }
  }
}

// A cell value at the face, q - t . g (t the offset from the face centroid
// to the cell centroid), as three fused multiply-adds.
__device__ __forceinline__ double reconstruct(double q, const double t[3], const double* g) {
  return fma(-t[2], g[2], fma(-t[1], g[1], fma(-t[0], g[0], q)));
}

template <int EX, int EY, int EZ>
__device__ __forceinline__ double edot(const double* g) {
  // e . g for a lattice direction with components in {-1, 0, 1}
  double s = 0.0;
  if (EX) s = EX > 0 ? g[0] : -g[0];
  if (EY) s = EY > 0 ? s + g[1] : s - g[1];
  if (EZ) s = EZ > 0 ? s + g[2] : s - g[2];
  return s;
}

// Branch of a lattice pair from s = e . n (see face_moments), as two bits.
// FL = 1 (the CPU Solver, Solver.cpp:840-1274) has no dead band: s == 0 takes
// both nodes from the owner side (3).
template <int EX, int EY, int EZ, int FL>
__device__ __forceinline__ unsigned pair_side(const double n[3], double d1) {
  const double s = (EX ? (EX > 0 ? n[0] : -n[0]) : 0.0) + (EY ? (EY > 0 ? n[1] : -n[1]) : 0.0) +
                   (EZ ? (EZ > 0 ? n[2] : -n[2]) : 0.0);
  if (FL == 1) return s > 0.0 ? 1u : (s < 0.0 ? 2u : 3u);
  return s > d1 ? 1u : (s < -d1 ? 2u : 0u);
}

// The interface moments of a face, in units of cD (below):
//   R = sum_k feq_k, m = sum_k e_k feq_k, P = sum_k e_k e_k^T feq_k (xx, yy, zz,
//   xy, xz, yz) over the 15 lattice nodes (populate_lattice_macros and
// populate_feq, LBFS.cu:330-1038). Node k sits at x_f - e_k dt_s; of the
// opposite pair (e, -e), s = e . n > d1 takes node e from the owner side and
// -e from the neighbour side, s < -d1 the reverse, and otherwise both come
// from the face average with averaged gradients (the +-0.001 dt dead band,
// LBFS.cu:353-354); `sides` holds pair_side of the seven pairs, two bits each.
// Faces are sorted by these bits, so the branches are uniform across almost
// every warp.
//
// The kernels that call this are bound by the FP64 pipe and the latency of
// their gathers, so the sum is arranged for the fewest FP64 instructions
// (298 per face on tetrahedra, 372-375 with a separate evaluation per
// node; k_flux on the 256x128x128 channel 487 -> 447 us, on 1.57 M tetrahedra
// 155 -> 148 us):
//  - A side's field value at a diagonal node is (s -+ dt gz) -+ dt (gx +- gy):
//    the first term is the z-axis node's value, the second bracket is shared
//    by two nodes, so the four diagonal values cost one FMA each once (s, gx,
//    gy, gz) has become (s - dt gz, s + dt gz, gx + gy, gx - gy) in place.
//  - feq = w rho (1 + 3 e.u + c45 (e.u)^2 - c15 u^2), c15 = 1.5 / gamma, c45 =
//    3 c15, is evaluated as w c15 rho (k0 - u^2 + e.u (k1 + 3 e.u)), k0 = 1 /
//    c15, k1 = 3 / c15: no scaled velocities, and on an axis node
//    3 u_n^2 - u^2 = 2 u_n^2 - the other two squares. The factor cD = c15 / 72
//    of the diagonal class is left out of all sums (flux_of_moments puts it in);
//    axis nodes weigh 8, the centre 16.
//  - The diagonal pairs' sums and differences go through the 4-point
//    Walsh-Hadamard sums two at a time instead of into seven accumulators each.
//
// The small terms of a node's bracket are summed before k0 is added (centre and
// axis nodes, 70 of the 72 parts): one rounding at its size instead of three.
//
// si, sn: owner- and neighbour-side values at the face, sc their mean, each
// (rho, u, v, w); g1, g2 the gradients [4 fields][3] (transformed in place).
template <int AX, int FL>
__device__ __forceinline__ void axis_pair(const double k0, const double k1, const double dt,
                                          const unsigned side, const double si[4],
                                          const double sn[4], const double sc[4],
                                          const double g1[12], const double g2[12], double& sum,
                                          double& dif) {
  double qa[4], qb[4];
  if (side == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(-g1[3 * f + AX], dt, si[f]);
      qb[f] = fma(g2[3 * f + AX], dt, sn[f]);
    }
  } else if (side == 2) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(-g2[3 * f + AX], dt, sn[f]);
      qb[f] = fma(g1[3 * f + AX], dt, si[f]);
    }
  } else if (FL == 1) {  // side 3: both nodes from the owner side
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(-g1[3 * f + AX], dt, si[f]);
      qb[f] = fma(g1[3 * f + AX], dt, si[f]);
    }
  } else {
    const double hdt = __dmul_rn(0.5, dt);
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const double e = __dadd_rn(g1[3 * f + AX], g2[3 * f + AX]);
      qa[f] = fma(-e, hdt, sc[f]);
      qb[f] = fma(e, hdt, sc[f]);
    }
  }
  constexpr int N = 1 + AX, T1 = 1 + (AX + 1) % 3, T2 = 1 + (AX + 2) % 3;
  const double ua = fma(qa[T1], qa[T1], __dmul_rn(qa[T2], qa[T2]));
  const double ub = fma(qb[T1], qb[T1], __dmul_rn(qb[T2], qb[T2]));
  const double ta = __dadd_rn(k0, fma(qa[N], fma(2.0, qa[N], k1), -ua));
  const double tb = __dadd_rn(k0, fma(qb[N], fma(2.0, qb[N], -k1), -ub));
  const double fb = __dmul_rn(qb[0], tb);
  sum = fma(qa[0], ta, fb);
  dif = fma(qa[0], ta, -fb);
}

// One diagonal pair (EX, EY, EZ), EZ = 1 or (1, 1, -1): zp, zm the sides'
// values s -+ dt gz, h the bracket gx + EX EY gy of each side.
template <int EX, int EY, int EZ, int FL>
__device__ __forceinline__ void diag_pair(const double k0, const double k1, const double dt,
                                          const unsigned side, const double z1p[4],
                                          const double z1m[4], const double z2p[4],
                                          const double z2m[4], const double g1[12],
                                          const double g2[12], double& sum, double& dif) {
  constexpr int HH = EX * EY > 0 ? 0 : 1;
  const double* a1 = EZ > 0 ? z1p : z1m;  // value at +e without the x, y part
  const double* b1 = EZ > 0 ? z1m : z1p;  // and at -e
  const double* a2 = EZ > 0 ? z2p : z2m;
  const double* b2 = EZ > 0 ? z2m : z2p;
  const double da = EX > 0 ? -dt : dt, db = EX > 0 ? dt : -dt;
  double qa[4], qb[4];
  if (side == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(da, g1[3 * f + HH], a1[f]);
      qb[f] = fma(db, g2[3 * f + HH], b2[f]);
    }
  } else if (side == 2) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(da, g2[3 * f + HH], a2[f]);
      qb[f] = fma(db, g1[3 * f + HH], b1[f]);
    }
  } else if (FL == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fma(da, g1[3 * f + HH], a1[f]);
      qb[f] = fma(db, g1[3 * f + HH], b1[f]);
    }
  } else {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = __dmul_rn(0.5, __dadd_rn(fma(da, g1[3 * f + HH], a1[f]),
                                       fma(da, g2[3 * f + HH], a2[f])));
      qb[f] = __dmul_rn(0.5, __dadd_rn(fma(db, g1[3 * f + HH], b1[f]),
                                       fma(db, g2[3 * f + HH], b2[f])));
    }
  }
  const double eua = edot<EX, EY, EZ>(qa + 1), eub = edot<-EX, -EY, -EZ>(qb + 1);
  const double ta = fma(eua, fma(3.0, eua, k1),
                        fma(-qa[1], qa[1], fma(-qa[2], qa[2], fma(-qa[3], qa[3], k0))));
  const double tb = fma(eub, fma(3.0, eub, k1),
                        fma(-qb[1], qb[1], fma(-qb[2], qb[2], fma(-qb[3], qb[3], k0))));
  const double fb = __dmul_rn(qb[0], tb);
  sum = fma(qa[0], ta, fb);
  dif = fma(qa[0], ta, -fb);
}

template <int FL>
__device__ __forceinline__ void face_moments(const double k0, const double k1, const double dt,
                                             const unsigned sides, double si[4], double sn[4],
                                             const double sc[4], double g1[12], double g2[12],
                                             double& R, double m[3], double P[6]) {
  // centre node: e = 0, weight 16
  const double u2 = fma(sc[3], sc[3], fma(sc[2], sc[2], __dmul_rn(sc[1], sc[1])));
  const double cen = __dmul_rn(sc[0], __dadd_rn(k0, -u2));
  double ax, ay, az, dx, dy, dz;
  axis_pair<0, FL>(k0, k1, dt, sides & 3, si, sn, sc, g1, g2, ax, dx);
  axis_pair<1, FL>(k0, k1, dt, sides >> 2 & 3, si, sn, sc, g1, g2, ay, dy);
  axis_pair<2, FL>(k0, k1, dt, sides >> 4 & 3, si, sn, sc, g1, g2, az, dz);
  const double axis = __dadd_rn(__dadd_rn(fma(2.0, cen, ax), ay), az);
  // (s, gx, gy, gz) -> (s - dt gz, s + dt gz, gx + gy, gx - gy); s - dt gz in
  // si / sn, s + dt gz in the `z1m` and `z2m`
  double z1m[4], z2m[4];
#pragma unroll
  for (int f = 0; f < 4; f++) {
    z1m[f] = fma(g1[3 * f + 2], dt, si[f]);
    si[f] = fma(-g1[3 * f + 2], dt, si[f]);
    z2m[f] = fma(g2[3 * f + 2], dt, sn[f]);
    sn[f] = fma(-g2[3 * f + 2], dt, sn[f]);
    const double s1 = __dadd_rn(g1[3 * f], g1[3 * f + 1]), r1 = __dadd_rn(g1[3 * f], -g1[3 * f + 1]);
    const double s2 = __dadd_rn(g2[3 * f], g2[3 * f + 1]), r2 = __dadd_rn(g2[3 * f], -g2[3 * f + 1]);
    g1[3 * f] = s1;
    g1[3 * f + 1] = r1;
    g2[3 * f] = s2;
    g2[3 * f + 1] = r2;
  }
  double s1, s2, d1, d2;
  diag_pair<1, 1, 1, FL>(k0, k1, dt, sides >> 6 & 3, si, z1m, sn, z2m, g1, g2, s1, d1);
  diag_pair<1, 1, -1, FL>(k0, k1, dt, sides >> 8 & 3, si, z1m, sn, z2m, g1, g2, s2, d2);
  const double sa = __dadd_rn(s1, s2), sb = __dadd_rn(s1, -s2);
  const double pa = __dadd_rn(d1, d2), pb = __dadd_rn(d1, -d2);
  diag_pair<1, -1, 1, FL>(k0, k1, dt, sides >> 10 & 3, si, z1m, sn, z2m, g1, g2, s1, d1);
  diag_pair<-1, 1, 1, FL>(k0, k1, dt, sides >> 12 & 3, si, z1m, sn, z2m, g1, g2, s2, d2);
  const double se = __dadd_rn(s1, s2), sf = __dadd_rn(s1, -s2);
  const double pe = __dadd_rn(d1, d2), pf = __dadd_rn(d1, -d2);
  const double D = __dadd_rn(sa, se);
  R = fma(8.0, axis, D);
  P[0] = fma(8.0, ax, D);
  P[1] = fma(8.0, ay, D);
  P[2] = fma(8.0, az, D);
  P[3] = __dadd_rn(sa, -se);
  P[4] = __dadd_rn(sb, sf);
  P[5] = __dadd_rn(sb, -sf);
  m[0] = fma(8.0, dx, __dadd_rn(pa, pf));
  m[1] = fma(8.0, dy, __dadd_rn(pa, -pf));
  m[2] = fma(8.0, dz, __dadd_rn(pb, pe));
}

// Flux of one face (calc_face_flux, LBFS.cu:1592-1710 and
// calculate_flux_at_interface, LBFS.cu:1042-1223), in closed form:
//   rho_I = sum_k feq_k(lattice), m = sum_k e_k feq_k(lattice), u_I = m / rho_I
//   f_k = feq_k(rho_I, u_I) - tau (feq_k(rho_I, u_I) - feq_k(lattice)),
//   tau = 3 nu / (dt_s gamma)
// whose moments are, exactly (D3Q15 equilibrium moments are isotropic):
//   sum e f = m
//   sum e e^T f = (1 - tau) (rho_I / 3 I + m m^T / (rho_I gamma)) + tau P_lattice
// The face flux is (momentum, mass) = ((sum e e^T f) n, (sum e f) . n) A, summed as
//   A p n + (1 - tau) A m (m . n) / (rho_I gamma) + tau A (P - p I) n,  p = rho_I / 3,
// so that the pressure, the largest term by far, is rounded twice and goes
// through none of the factors that are a face's own, omA = (1 - tau) A cD and tA =
// tau A cD: what those lose by rounding is the same in every step, and as a part
// of the pressure it was an imbalance around each cell (64^3 jittered hexes in
// tetrahedra, error of 40 steps against plain 64-bit sums: 3.3e-14 with the
// pressure in omA and tA, 2.3e-14 so, at the same time).
// A boundary face (neighbour > n_cells in the reference) takes both sides from
// the boundary value and all gradients from the ghost (LBFS.cu:356-401).
__device__ __forceinline__ d4 flux_of_moments(const KernelArgs& a, const double R,
                                              const double m[3], const double P[6],
                                              const double n[3], const double A,
                                              const double omA, const double tA) {
  const double mn = fma(m[2], n[2], fma(m[1], n[1], __dmul_rn(m[0], n[0])));
  const double D[3] = {fma(-1.0 / 3.0, R, P[0]), fma(-1.0 / 3.0, R, P[1]), fma(-1.0 / 3.0, R, P[2])};
  const double Dn[3] = {fma(P[4], n[2], fma(P[3], n[1], __dmul_rn(D[0], n[0]))),
                        fma(P[5], n[2], fma(D[1], n[1], __dmul_rn(P[3], n[0]))),
                        fma(D[2], n[2], fma(P[5], n[1], __dmul_rn(P[4], n[0])))};
  const double am = __dmul_rn(omA, __dmul_rn(__ddiv_rn(mn, R), a.pg));
  const double Ap = __dmul_rn(A, __dmul_rn(R, a.eq_cd3));
  d4 out;
  out.x = fma(Ap, n[0], fma(tA, Dn[0], __dmul_rn(am, m[0])));
  out.y = fma(Ap, n[1], fma(tA, Dn[1], __dmul_rn(am, m[1])));
  out.z = fma(Ap, n[2], fma(tA, Dn[2], __dmul_rn(am, m[2])));
  out.w = __dmul_rn(__dmul_rn(mn, a.eq_cd), A);
  return out;
}

// The seven branch decisions of a face (face_moments' sides).
template <int FL>
__device__ __forceinline__ unsigned face_sides(const double n[3], double dt) {
  const double d1 = 0.001 * dt;
  return pair_side<1, 0, 0, FL>(n, d1) | pair_side<0, 1, 0, FL>(n, d1) << 2 |
         pair_side<0, 0, 1, FL>(n, d1) << 4 | pair_side<1, 1, 1, FL>(n, d1) << 6 |
         pair_side<1, 1, -1, FL>(n, d1) << 8 | pair_side<1, -1, 1, FL>(n, d1) << 10 |
         pair_side<-1, 1, 1, FL>(n, d1) << 12;
}

// A face's side values (si, sn, sc) and the gradients its nodes use (g1, g2)
// from its cells: qo and g1 the owner's state and gradient; internal faces
// qn and g2 the neighbour's; boundary faces (b >= 0 the device boundary
// index) build theirs from the boundary records.
__device__ __forceinline__ void interior_sides(const double t1[3], const double t2[3],
                                                    const d4& qo, const d4& qn,
                                                    const double g1[12], const double g2[12],
                                                    double si[4], double sn[4], double sc[4]) {
  const double qov[4] = {qo.w, qo.x, qo.y, qo.z}, qnv[4] = {qn.w, qn.x, qn.y, qn.z};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    si[k] = reconstruct(qov[k], t1, g1 + 3 * k);
    sn[k] = reconstruct(qnv[k], t2, g2 + 3 * k);
    sc[k] = __dmul_rn(__dadd_rn(si[k], sn[k]), 0.5);
  }
}

// Records of faces along a coordinate axis: one component of n, t1 and t2 is
// nonzero and the branch bits are those of n = +e_AX. Their kind, 1 + AX, sits
// above the branch bits of the compact layout's records (face_kind; 0: general
// faces and n = -e, which a box has on its boundary only), and the kernels
// take a branch per axis in which the seven lattice branches are resolved at
// compile time and the products with the zero components are left out: the
// same value for every finite state. On the 256x128x128 channel k_flux 443 -> 424
// us, k_flux32 255 -> 228 us. The march kernel stays with the general path: its
// blocks go through the code once per stage, and three more copies of it cost
// more than they save there (32^3 cavity 40 -> 43 us per step).
constexpr int kKindShift = 14;
template <int FL, int AX>
__host__ __device__ constexpr unsigned axis_sides() {
  unsigned s = 0;
  const int e[7][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 1}, {1, 1, -1}, {1, -1, 1}, {-1, 1, 1}};
  for (int p = 0; p < 7; p++)
    s |= (e[p][AX] > 0 ? 1u : e[p][AX] < 0 ? 2u : FL == 1 ? 3u : 0u) << (2 * p);
  return s;
}
template <int FL>
__device__ __forceinline__ unsigned face_kind(const d4& f0, const d4& f1, const d4& f2,
                                              unsigned sides) {
  const double n[3] = {f0.x, f0.y, f0.z}, t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
  const unsigned want[3] = {axis_sides<FL, 0>(), axis_sides<FL, 1>(), axis_sides<FL, 2>()};
  for (int x = 0; x < 3; x++) {
    bool ok = sides == want[x];
    for (int c = 0; c < 3; c++)
      if (c != x) ok = ok && n[c] == 0.0 && t1[c] == 0.0 && t2[c] == 0.0;
    if (ok) return 1u + x;
  }
  return 0u;
}

// An internal face of kind 1 + AX: its flux from t1 = t1d e, t2 = t2d e, n = nd e.
template <int FL, int AX>
__device__ __forceinline__ d4 axis_flux(const KernelArgs& a, const double dt, const double t1d,
                                        const double t2d, const double nd, const double A,
                                        const double omA, const double tA, const d4& qo,
                                        const d4& qn, double g1[12], double g2[12]) {
  const double qov[4] = {qo.w, qo.x, qo.y, qo.z}, qnv[4] = {qn.w, qn.x, qn.y, qn.z};
  double si[4], sn[4], sc[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    si[k] = fma(-t1d, g1[3 * k + AX], qov[k]);
    sn[k] = fma(-t2d, g2[3 * k + AX], qnv[k]);
    sc[k] = __dmul_rn(__dadd_rn(si[k], sn[k]), 0.5);
  }
  double R, m[3], P[6];
  face_moments<FL>(a.eq_k0, a.eq_k1, dt, axis_sides<FL, AX>(), si, sn, sc, g1, g2, R, m, P);
  const double mn = __dmul_rn(m[AX], nd);
  // the AX column of P (xx, yy, zz, xy, xz, yz)
  constexpr int C0 = AX == 0 ? 0 : AX == 1 ? 3 : 4, C1 = AX == 0 ? 3 : AX == 1 ? 1 : 5,
                C2 = AX == 0 ? 4 : AX == 1 ? 5 : 2;
  const double Pc[3] = {P[C0], P[C1], P[C2]};
  const double am = __dmul_rn(omA, __dmul_rn(__ddiv_rn(mn, R), a.pg));
  const double Ap = __dmul_rn(A, __dmul_rn(R, a.eq_cd3));
  double out[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double Dn = __dmul_rn(c == AX ? fma(-1.0 / 3.0, R, Pc[c]) : Pc[c], nd);
    out[c] = fma(tA, Dn, __dmul_rn(am, m[c]));
    if (c == AX) out[c] = fma(Ap, nd, out[c]);
  }
  return d4{out[0], out[1], out[2], __dmul_rn(__dmul_rn(mn, a.eq_cd), A)};
}

template <int FL>
__device__ __forceinline__ void boundary_sides(const KernelArgs& a, const int b,
                                                    const double t1[3], const double t2[3],
                                                    const d4& qo, double g1[12], double g2[12],
                                                    double si[4], double sn[4], double sc[4]) {
  const d4 bv = ld4(a.bc0, b), tgt = ld4(a.bc1, b), dd = ld4(a.bc2, b), nm = ld4(a.bc3, b);
  const int types = (int)nm.w;
  ghost_grad<FL>(qo, g1, bv, dd, nm, types, g2);
  if (b == a.quirk_b) {
    // The reference tests neighbour > n_cells (LBFS.cu:356), so its first
    // ghost (index n_cells) goes through the interior branch with the ghost
    // state and gradient as the neighbour's.
    interior_sides(t1, t2, qo, ghost_state<FL>(qo, tgt, types), g1, g2, si, sn, sc);
    return;
  }
  const double qov[4] = {qo.w, qo.x, qo.y, qo.z};
  const int rt = types & 0xff, vt = types >> 8;
  const double bvv[4] = {bv.w, bv.x, bv.y, bv.z};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // FL = 1 (populate_lattice_macros, Solver.cpp:862-904): rho 1 and
    // velocity 1 the value, velocity 8 (u, 0, w) of the owner, otherwise
    // extrapolated with the ghost gradient
    const bool dirichlet = (k == 0) ? (rt == 1) : (FL == 1 ? vt == 1 : vt != 2);
    const double ext = reconstruct(qov[k], t1, g2 + 3 * k);
    sc[k] = dirichlet ? bvv[k] : (FL == 1 && k > 0 && vt == 8) ? (k == 2 ? 0.0 : qov[k]) : ext;
    si[k] = sc[k];
    sn[k] = sc[k];
  }
  // FL = 0: the ghost gradient on both sides (LBFS.cu:398-401); FL = 1
  // keeps the owner's on the owner side
  if (FL == 0) {
#pragma unroll
    for (int k = 0; k < 12; k++) g1[k] = g2[k];
  }
}

// The flux from the side values. r indexes the face's records: the compact
// tables with CR, else the per-face arrays. n, A and the area factors are
// read again here (L1 hits) rather than held in registers through the pairs.
template <int FL, bool CR>
__device__ __forceinline__ d4 face_flux(const KernelArgs& a, const int r, const unsigned sides,
                                        const double dt, double si[4], double sn[4],
                                        const double sc[4], double g1[12], double g2[12]) {
  double R, m[3], P[6];
  face_moments<FL>(a.eq_k0, a.eq_k1, dt, sides, si, sn, sc, g1, g2, R, m, P);
  const d4 g0 = ld4(launder(CR ? a.frec0 : a.face0), r);
  const double n[3] = {g0.x, g0.y, g0.z};
  const double A = g0.w;
  double omA, tA;
  if (CR) {
    const double2 w = __ldg(reinterpret_cast<const double2*>(a.frec_relax) + r);
    omA = w.x;
    tA = w.y;
  } else {
    const double tau = __ldg(static_cast<const double*>(launder(a.face2)) + 4LL * r + 3);
    const double cA = __dmul_rn(A, a.eq_cd);
    omA = __dmul_rn(__dadd_rn(1.0, -tau), cA);
    tA = __dmul_rn(tau, cA);
  }
  return flux_of_moments(a, R, m, P, n, A, omA, tA);
}

// One cell's RK stage (time_integration, LBFS.cu:1457-1521) from its residual R
// (u, v, w, rho): the stage state q and the accumulator. t0 is the step's
// start, t1 the running accumulator; at a step boundary they are equal (the
// next step starts from the accumulator, Solver_gpu.cu:671), so stage 0 takes
// t0 for both and stage 3, whose state is the accumulator's, does not need t0.
template <int RK>
__device__ __forceinline__ void rk_stage(const double dt, const d4& t0, const d4& t1,
                                         const double R[4], d4& q, d4& acc) {
  constexpr double alpha = (RK == 0 || RK == 3) ? 1.0 : 0.5;
  constexpr double beta = (RK == 0 || RK == 3) ? (1.0 / 6.0) : (1.0 / 3.0);
  const double bdt = __dmul_rn(dt, beta);
  const d4& b = RK == 0 ? t0 : t1;
  acc = d4{fma(R[0], bdt, b.x), fma(R[1], bdt, b.y), fma(R[2], bdt, b.z), fma(R[3], bdt, b.w)};
  if (RK == 3) {
    q = d4{__ddiv_rn(acc.x, acc.w), __ddiv_rn(acc.y, acc.w), __ddiv_rn(acc.z, acc.w), acc.w};
  } else {
    const double adt = __dmul_rn(dt, alpha), f = fma(R[3], adt, t0.w);
    q = d4{__ddiv_rn(fma(R[0], adt, t0.x), f), __ddiv_rn(fma(R[1], adt, t0.y), f),
           __ddiv_rn(fma(R[2], adt, t0.z), f), f};
  }
}

}  // namespace
}  // namespace plfbs
