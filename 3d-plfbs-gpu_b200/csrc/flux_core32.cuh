// ---------------------------------------------------------------------------
// Flux core of the FP32 deviation form (see kernels_fp32.cu for its variables):
// record accesses and per-face arithmetic shared by the face kernels
// (kernels_fp32.cu) and the march kernel (march.cu, tiles.cu), with explicit
// roundings as in flux_core.cuh, so that both compute the same bits.
// ---------------------------------------------------------------------------
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "flux_core.cuh"
#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

struct __align__(16) f4 {
  float x, y, z, w;
};

__device__ __forceinline__ f4 ldf(const void* base, long long i) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(base) + i);
  return f4{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ f4 ldf_rw(const void* base, long long i) {
  const float4 v = reinterpret_cast<const float4*>(base)[i];
  return f4{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ void stf(void* base, long long i, const f4& v) {
  reinterpret_cast<float4*>(base)[i] = make_float4(v.x, v.y, v.z, v.w);
}

// Ghost state in deviation units (the same affine rules as the FP64 path).
__device__ __forceinline__ f4 ghost_state32(const f4& q, const f4& tgt, int types) {
  const int rt = types & 0xff, vt = types >> 8;
  f4 g;
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

__device__ __forceinline__ void load_grad32(const void* base, int c, float g[12]) {
  const f4 a0 = ldf(base, 3LL * c), a1 = ldf(base, 3LL * c + 1), a2 = ldf(base, 3LL * c + 2);
  g[0] = a0.x; g[1] = a0.y; g[2] = a0.z; g[3] = a0.w;
  g[4] = a1.x; g[5] = a1.y; g[6] = a1.z; g[7] = a1.w;
  g[8] = a2.x; g[9] = a2.y; g[10] = a2.z; g[11] = a2.w;
}

__device__ __forceinline__ void ghost_grad32(const f4& q, const float go[12], const f4& bv,
                                             const f4& dd, const f4& nm, int types, float g[12]) {
  const int rt = types & 0xff, vt = types >> 8;
  const float dir[3] = {dd.x, dd.y, dd.z}, m[3] = {nm.x, nm.y, nm.z};
  const float dq[4] = {2.0f * (bv.w - q.w), 2.0f * (bv.x - q.x), 2.0f * (bv.y - q.y),
                       2.0f * (bv.z - q.z)};
#pragma unroll
  for (int f = 0; f < 4; f++) {
    const bool dirichlet = (f == 0) ? (rt == 1) : (vt != 2);
#pragma unroll
    for (int c = 0; c < 3; c++)
      g[3 * f + c] = dirichlet ? dq[f] / dd.w * dir[c] : go[3 * f + c] * m[c];
  }
}

// Branch bits of a face's seven lattice pairs (pair_side and face_sides of
// flux_core.cuh in FP32, GPU flavour), d1 = 0.001 dt.
__device__ __forceinline__ unsigned face_sides32(float nx, float ny, float nz, float d1) {
  const float s[7] = {nx,
                      ny,
                      nz,
                      __fadd_rn(__fadd_rn(nx, ny), nz),
                      __fadd_rn(__fadd_rn(nx, ny), -nz),
                      __fadd_rn(__fadd_rn(nx, -ny), nz),
                      __fadd_rn(__fadd_rn(-nx, ny), nz)};
  unsigned sides = 0;
#pragma unroll
  for (int p = 0; p < 7; p++) sides |= (s[p] > d1 ? 1u : (s[p] < -d1 ? 2u : 0u)) << (2 * p);
  return sides;
}

// Interface moments as face_moments (flux_core.cuh), of the deviation part of
// the equilibrium, w [drho + rho U phi], in units of cD = c / 72 with c = 1.5 U^2
// / gamma:
//   f / (w c) = k0 drho + rho (e.u' (k1 + 3 e.u') - u'^2),  k0 = 1 / c,
//   k1 = 2 gamma / U.
struct Eq32 {
  float k0, k1, rho0;
};

__device__ __forceinline__ float edotf(int ex, int ey, int ez, const float* g) {
  const float s = ey > 0 ? __fadd_rn(ex > 0 ? g[0] : -g[0], g[1])
                         : __fadd_rn(ex > 0 ? g[0] : -g[0], -g[1]);
  return ez > 0 ? __fadd_rn(s, g[2]) : __fadd_rn(s, -g[2]);
}

__device__ __forceinline__ float node_value(const Eq32& k, const float q[4], float t) {
  return fmaf(__fadd_rn(k.rho0, q[0]), t, __fmul_rn(k.k0, q[0]));
}

template <int AX>
__device__ __forceinline__ void axis_pair32(const Eq32& k, const float dt, const unsigned side,
                                            const float si[4], const float sn[4],
                                            const float sc[4], const float g1[12],
                                            const float g2[12], float& sum, float& dif) {
  float qa[4], qb[4];
  if (side == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fmaf(-g1[3 * f + AX], dt, si[f]);
      qb[f] = fmaf(g2[3 * f + AX], dt, sn[f]);
    }
  } else if (side == 2) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fmaf(-g2[3 * f + AX], dt, sn[f]);
      qb[f] = fmaf(g1[3 * f + AX], dt, si[f]);
    }
  } else {
    const float hdt = __fmul_rn(0.5f, dt);
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const float e = __fadd_rn(g1[3 * f + AX], g2[3 * f + AX]);
      qa[f] = fmaf(-e, hdt, sc[f]);
      qb[f] = fmaf(e, hdt, sc[f]);
    }
  }
  constexpr int N = 1 + AX, T1 = 1 + (AX + 1) % 3, T2 = 1 + (AX + 2) % 3;
  const float ta = fmaf(qa[N], fmaf(2.0f, qa[N], k.k1), -fmaf(qa[T1], qa[T1], __fmul_rn(qa[T2], qa[T2])));
  const float tb = fmaf(qb[N], fmaf(2.0f, qb[N], -k.k1), -fmaf(qb[T1], qb[T1], __fmul_rn(qb[T2], qb[T2])));
  const float fa = node_value(k, qa, ta), fb = node_value(k, qb, tb);
  sum = __fadd_rn(fa, fb);
  dif = __fadd_rn(fa, -fb);
}

template <int EX, int EY, int EZ>
__device__ __forceinline__ void diag_pair32(const Eq32& k, const float dt, const unsigned side,
                                            const float z1p[4], const float z1m[4],
                                            const float z2p[4], const float z2m[4],
                                            const float g1[12], const float g2[12], float& sum,
                                            float& dif) {
  constexpr int HH = EX * EY > 0 ? 0 : 1;
  const float* a1 = EZ > 0 ? z1p : z1m;
  const float* b1 = EZ > 0 ? z1m : z1p;
  const float* a2 = EZ > 0 ? z2p : z2m;
  const float* b2 = EZ > 0 ? z2m : z2p;
  const float da = EX > 0 ? -dt : dt, db = EX > 0 ? dt : -dt;
  float qa[4], qb[4];
  if (side == 1) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fmaf(da, g1[3 * f + HH], a1[f]);
      qb[f] = fmaf(db, g2[3 * f + HH], b2[f]);
    }
  } else if (side == 2) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = fmaf(da, g2[3 * f + HH], a2[f]);
      qb[f] = fmaf(db, g1[3 * f + HH], b1[f]);
    }
  } else {
#pragma unroll
    for (int f = 0; f < 4; f++) {
      qa[f] = __fmul_rn(0.5f, __fadd_rn(fmaf(da, g1[3 * f + HH], a1[f]),
                                        fmaf(da, g2[3 * f + HH], a2[f])));
      qb[f] = __fmul_rn(0.5f, __fadd_rn(fmaf(db, g1[3 * f + HH], b1[f]),
                                        fmaf(db, g2[3 * f + HH], b2[f])));
    }
  }
  const float eua = edotf(EX, EY, EZ, qa + 1), eub = edotf(-EX, -EY, -EZ, qb + 1);
  const float ua = fmaf(qa[3], qa[3], fmaf(qa[2], qa[2], __fmul_rn(qa[1], qa[1])));
  const float ub = fmaf(qb[3], qb[3], fmaf(qb[2], qb[2], __fmul_rn(qb[1], qb[1])));
  const float fa = node_value(k, qa, fmaf(eua, fmaf(3.0f, eua, k.k1), -ua));
  const float fb = node_value(k, qb, fmaf(eub, fmaf(3.0f, eub, k.k1), -ub));
  sum = __fadd_rn(fa, fb);
  dif = __fadd_rn(fa, -fb);
}

__device__ __forceinline__ void face_moments32(const Eq32& k, const float dt, const unsigned sides,
                                               float si[4], float sn[4], const float sc[4],
                                               float g1[12], float g2[12], float& R, float m[3],
                                               float P[6]) {
  // centre node: e = 0, weight 16
  const float cen = node_value(
      k, sc, -fmaf(sc[3], sc[3], fmaf(sc[2], sc[2], __fmul_rn(sc[1], sc[1]))));
  float ax, ay, az, dx, dy, dz;
  axis_pair32<0>(k, dt, sides & 3, si, sn, sc, g1, g2, ax, dx);
  axis_pair32<1>(k, dt, sides >> 2 & 3, si, sn, sc, g1, g2, ay, dy);
  axis_pair32<2>(k, dt, sides >> 4 & 3, si, sn, sc, g1, g2, az, dz);
  const float axis = __fadd_rn(__fadd_rn(fmaf(2.0f, cen, ax), ay), az);
  float z1m[4], z2m[4];
#pragma unroll
  for (int f = 0; f < 4; f++) {
    z1m[f] = fmaf(g1[3 * f + 2], dt, si[f]);
    si[f] = fmaf(-g1[3 * f + 2], dt, si[f]);
    z2m[f] = fmaf(g2[3 * f + 2], dt, sn[f]);
    sn[f] = fmaf(-g2[3 * f + 2], dt, sn[f]);
    const float s1 = __fadd_rn(g1[3 * f], g1[3 * f + 1]), r1 = __fadd_rn(g1[3 * f], -g1[3 * f + 1]);
    const float s2 = __fadd_rn(g2[3 * f], g2[3 * f + 1]), r2 = __fadd_rn(g2[3 * f], -g2[3 * f + 1]);
    g1[3 * f] = s1;
    g1[3 * f + 1] = r1;
    g2[3 * f] = s2;
    g2[3 * f + 1] = r2;
  }
  float s1, s2, d1, d2;
  diag_pair32<1, 1, 1>(k, dt, sides >> 6 & 3, si, z1m, sn, z2m, g1, g2, s1, d1);
  diag_pair32<1, 1, -1>(k, dt, sides >> 8 & 3, si, z1m, sn, z2m, g1, g2, s2, d2);
  const float sa = __fadd_rn(s1, s2), sb = __fadd_rn(s1, -s2);
  const float pa = __fadd_rn(d1, d2), pb = __fadd_rn(d1, -d2);
  diag_pair32<1, -1, 1>(k, dt, sides >> 10 & 3, si, z1m, sn, z2m, g1, g2, s1, d1);
  diag_pair32<-1, 1, 1>(k, dt, sides >> 12 & 3, si, z1m, sn, z2m, g1, g2, s2, d2);
  const float se = __fadd_rn(s1, s2), sf = __fadd_rn(s1, -s2);
  const float pe = __fadd_rn(d1, d2), pf = __fadd_rn(d1, -d2);
  const float D = __fadd_rn(sa, se);
  R = fmaf(8.0f, axis, D);
  P[0] = fmaf(8.0f, ax, D);
  P[1] = fmaf(8.0f, ay, D);
  P[2] = fmaf(8.0f, az, D);
  P[3] = __fadd_rn(sa, -se);
  P[4] = __fadd_rn(sb, sf);
  P[5] = __fadd_rn(sb, -sf);
  m[0] = fmaf(8.0f, dx, __fadd_rn(pa, pf));
  m[1] = fmaf(8.0f, dy, __fadd_rn(pa, -pf));
  m[2] = fmaf(8.0f, dz, __fadd_rn(pb, pe));
}

// A cell value at the face, q - t . g.
__device__ __forceinline__ float reconstruct32(float q, const float t[3], const float* g) {
  return __fadd_rn(q, -fmaf(t[2], g[2], fmaf(t[1], g[1], __fmul_rn(t[0], g[0]))));
}

// Side values of an internal and of a boundary face (interior_sides and
// boundary_sides of flux_core.cuh, GPU flavour).
__device__ __forceinline__ void interior_sides32(const float t1[3], const float t2[3],
                                                 const f4& qo, const f4& qn, const float g1[12],
                                                 const float g2[12], float si[4], float sn[4],
                                                 float sc[4]) {
  const float qov[4] = {qo.w, qo.x, qo.y, qo.z}, qnv[4] = {qn.w, qn.x, qn.y, qn.z};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    si[k] = reconstruct32(qov[k], t1, g1 + 3 * k);
    sn[k] = reconstruct32(qnv[k], t2, g2 + 3 * k);
    sc[k] = __fmul_rn(__fadd_rn(si[k], sn[k]), 0.5f);
  }
}

__device__ __forceinline__ void boundary_sides32(const KernelArgs& a, const int b,
                                                 const float t1[3], const float t2[3],
                                                 const f4& qo, float g1[12], float g2[12],
                                                 float si[4], float sn[4], float sc[4]) {
  const f4 bv = ldf(a.bc0, b), tgt = ldf(a.bc1, b), dd = ldf(a.bc2, b), nm = ldf(a.bc3, b);
  const int types = (int)nm.w;
  ghost_grad32(qo, g1, bv, dd, nm, types, g2);
  if (b == a.quirk_b) {  // interior branch, LBFS.cu:356
    interior_sides32(t1, t2, qo, ghost_state32(qo, tgt, types), g1, g2, si, sn, sc);
    return;
  }
  const float qov[4] = {qo.w, qo.x, qo.y, qo.z};
  const int rt = types & 0xff, vt = types >> 8;
  const float bvv[4] = {bv.w, bv.x, bv.y, bv.z};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool dirichlet = (k == 0) ? (rt == 1) : (vt != 2);
    sc[k] = dirichlet ? bvv[k] : reconstruct32(qov[k], t1, g2 + 3 * k);
    si[k] = sc[k];
    sn[k] = sc[k];
  }
#pragma unroll
  for (int k = 0; k < 12; k++) g1[k] = g2[k];
}

// Records of faces along a coordinate axis, as face_kind and axis_flux in
// flux_core.cuh.
__device__ __forceinline__ unsigned face_kind32(const f4& f0, const f4& f1, const f4& f2,
                                                unsigned sides) {
  const float n[3] = {f0.x, f0.y, f0.z}, t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
  const unsigned want[3] = {axis_sides<0, 0>(), axis_sides<0, 1>(), axis_sides<0, 2>()};
  for (int x = 0; x < 3; x++) {
    bool ok = sides == want[x];
    for (int c = 0; c < 3; c++)
      if (c != x) ok = ok && n[c] == 0.0f && t1[c] == 0.0f && t2[c] == 0.0f;
    if (ok) return 1u + x;
  }
  return 0u;
}

template <int AX>
__device__ __forceinline__ f4 axis_flux32(const KernelArgs& a, const float dt, const float t1d,
                                          const float t2d, const float nd, const float area,
                                          const float tau, const f4& qo, const f4& qn,
                                          float g1[12], float g2[12]) {
  const float qov[4] = {qo.w, qo.x, qo.y, qo.z}, qnv[4] = {qn.w, qn.x, qn.y, qn.z};
  float si[4], sn[4], sc[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    si[k] = __fadd_rn(qov[k], -__fmul_rn(t1d, g1[3 * k + AX]));
    sn[k] = __fadd_rn(qnv[k], -__fmul_rn(t2d, g2[3 * k + AX]));
    sc[k] = __fmul_rn(__fadd_rn(si[k], sn[k]), 0.5f);
  }
  const Eq32 k{a.eq32_k0, a.eq32_k1, a.rho0f};
  float R, m[3], P[6];
  face_moments32(k, dt, axis_sides<0, AX>(), si, sn, sc, g1, g2, R, m, P);
  const float mn = __fmul_rn(m[AX], nd);
  constexpr int C0 = AX == 0 ? 0 : AX == 1 ? 3 : 4, C1 = AX == 0 ? 3 : AX == 1 ? 1 : 5,
                C2 = AX == 0 ? 4 : AX == 1 ? 5 : 2;
  const float Pn[3] = {__fmul_rn(P[C0], nd), __fmul_rn(P[C1], nd), __fmul_rn(P[C2], nd)};
  const float cA = __fmul_rn(area, a.eq32_cd), sA = __fmul_rn(cA, a.inv_uref_f);
  const float omA = __fmul_rn(__fadd_rn(1.0f, -tau), sA), tA = __fmul_rn(tau, sA);
  const float mnr = __fdiv_rn(__fmul_rn(mn, a.eq32_pgcd), fmaf(a.eq32_cd, R, k.rho0));
  const float al = __fmul_rn(omA, mnr), be = __fmul_rn(omA, __fmul_rn(R, 1.0f / 3.0f));
  float out[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const float tp = __fmul_rn(tA, Pn[c]);
    out[c] = fmaf(al, m[c], c == AX ? fmaf(be, nd, tp) : tp);
  }
  return f4{out[0], out[1], out[2], __fmul_rn(mn, cA)};
}

// The face flux in deviation form: the rho0 / 3 n A part of the momentum flux
// left out, momentum divided by U (see kernels_fp32.cu).
__device__ __forceinline__ f4 face_flux32(const KernelArgs& a, const float n[3], const float area,
                                          const float tau, const unsigned sides, const float dt,
                                          float si[4], float sn[4], const float sc[4],
                                          float g1[12], float g2[12]) {
  const Eq32 k{a.eq32_k0, a.eq32_k1, a.rho0f};
  float R, m[3], P[6];
  face_moments32(k, dt, sides, si, sn, sc, g1, g2, R, m, P);
  const float mn = fmaf(m[2], n[2], fmaf(m[1], n[1], __fmul_rn(m[0], n[0])));
  const float Pn[3] = {fmaf(P[4], n[2], fmaf(P[3], n[1], __fmul_rn(P[0], n[0]))),
                       fmaf(P[5], n[2], fmaf(P[1], n[1], __fmul_rn(P[3], n[0]))),
                       fmaf(P[2], n[2], fmaf(P[5], n[1], __fmul_rn(P[4], n[0])))};
  // rho_I = rho0 + cD R; momentum terms carry cD A / U, the mass flux cD A
  const float cA = __fmul_rn(area, a.eq32_cd), sA = __fmul_rn(cA, a.inv_uref_f);
  const float omA = __fmul_rn(__fadd_rn(1.0f, -tau), sA), tA = __fmul_rn(tau, sA);
  const float mnr = __fdiv_rn(__fmul_rn(mn, a.eq32_pgcd), fmaf(a.eq32_cd, R, k.rho0));
  const float al = __fmul_rn(omA, mnr), be = __fmul_rn(omA, __fmul_rn(R, 1.0f / 3.0f));
  f4 out;
  out.x = fmaf(al, m[0], fmaf(be, n[0], __fmul_rn(tA, Pn[0])));
  out.y = fmaf(al, m[1], fmaf(be, n[1], __fmul_rn(tA, Pn[1])));
  out.z = fmaf(al, m[2], fmaf(be, n[2], __fmul_rn(tA, Pn[2])));
  out.w = __fmul_rn(mn, cA);
  return out;
}

// One cell's RK stage in deviation units (as rk_stage in flux_core.cuh).
template <int RK>
__device__ __forceinline__ void rk_stage32(const float dt, const float rho0, const f4& t0,
                                           const f4& t1, const float R[4], f4& q, f4& acc) {
  constexpr float alpha = (RK == 0 || RK == 3) ? 1.0f : 0.5f;
  constexpr float beta = (RK == 0 || RK == 3) ? (1.0f / 6.0f) : (1.0f / 3.0f);
  const float bdt = __fmul_rn(dt, beta);
  const f4& b = RK == 0 ? t0 : t1;
  acc = f4{fmaf(R[0], bdt, b.x), fmaf(R[1], bdt, b.y), fmaf(R[2], bdt, b.z),
           fmaf(R[3], bdt, b.w)};
  f4 f = acc;
  if (RK != 3) {
    const float adt = __fmul_rn(dt, alpha);
    f = f4{fmaf(R[0], adt, t0.x), fmaf(R[1], adt, t0.y), fmaf(R[2], adt, t0.z),
           fmaf(R[3], adt, t0.w)};
  }
  const float rho = __fadd_rn(rho0, f.w);
  q = f4{__fdiv_rn(f.x, rho), __fdiv_rn(f.y, rho), __fdiv_rn(f.z, rho), f.w};
}

}  // namespace
}  // namespace plfbs
