// The immersed body's nodes (immersed_boundary_method.cu:13-90, 161-190,
// 244-295, 299-375), once per time step before the RK stages, as device code of
// the IBM kernels and of the march kernel (march.cu); explicit roundings where
// a product meets a sum, so that both give the same bits.
#pragma once

#include "flux_core.cuh"
#include "flux_core32.cuh"
#include "ibm_spread.cuh"

namespace plfbs {
namespace {

__device__ __forceinline__ void stencil_origin(const KernelArgs& a, const double x[3],
                                               double r[3], int lo[3]) {
  r[0] = (x[0] - a.origin[0]) / a.ibm_dx;
  r[1] = fabs((x[1] - a.origin[1]) / a.ibm_dx);
  r[2] = fabs((x[2] - a.origin[2]) / a.ibm_dx);
#pragma unroll
  for (int c = 0; c < 3; c++) lo[c] = (int)round(r[c]) - 1;
}

// Eight threads per node, one per cell of its 2 x 2 x 2 stencil: each loads
// its cell's state, the node's velocity is the sum over the eight (xor
// butterfly, so every lane holds the same bits), every lane advances the node
// and forms its force, and the warp spreads its lanes' forces with one FP64
// atomic per distinct cell and component (spread_aggregated; nodes in the
// spatial order ibm_order). Lane 0 of a node writes the node's arrays. t is the
// thread's index over all nodes, whole warps at a time.
__device__ __forceinline__ void ibm_thread(const KernelArgs& a, const int t) {
  const int slot = t >> 3, sub = t & 7;
  const bool active = slot < a.N;
  const int nd = active ? __ldg(a.ibm_order + slot) : 0;
  const int xc = a.ibm_xc, yc = a.ibm_yc;
  double x[3] = {0.0, 0.0, 0.0}, r[3] = {0.0, 0.0, 0.0};
  int lo[3] = {0, 0, 0};
  if (active) {
#pragma unroll
    for (int c = 0; c < 3; c++) x[c] = a.node_x[3 * nd + c];
    stencil_origin(a, x, r, lo);
  }
  const int di = sub & 1, dj = (sub >> 1) & 1, dk = sub >> 2;
  double v[3] = {0.0, 0.0, 0.0};
  {
    const int ii = lo[0] + di, jj = lo[1] + dj, kk = lo[2] + dk;
    const long long cell = (long long)ii + (long long)jj * xc + (long long)kk * yc * xc;
    if (active && cell < a.C && cell >= 0) {  // the reference's linear-index check
      const double wx = 1 - fabs(ii + 0.5 - r[0]);
      const double wy = 1 - fabs(jj + 0.5 - r[1]);
      const double wz = 1 - fabs(kk + 0.5 - r[2]);
      const d4 q = ld4rw(a.state, a.ibm_map[cell]);
      v[0] = __dmul_rn(q.x * wx * wy * wz, a.ibm_inv_dx3);
      v[1] = __dmul_rn(q.y * wx * wy * wz, a.ibm_inv_dx3);
      v[2] = __dmul_rn(q.z * wx * wy * wz, a.ibm_inv_dx3);
    }
  }
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1)
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] += __shfl_xor_sync(full, v[c], o);
  const unsigned act = __ballot_sync(full, active);
  if (!active) return;
  double fn[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    x[c] = fma(v[c], a.dt, a.node_x0[3 * nd + c]);
    fn[c] = -a.ibm_area_k * (x[c] - a.node_ref[3 * nd + c]);
  }
  if (sub == 0) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      a.node_x[3 * nd + c] = x[c];
      a.node_x0[3 * nd + c] = x[c];
      a.node_vel[3 * nd + c] = v[c];
      a.node_force[3 * nd + c] = fn[c];
    }
  }
  stencil_origin(a, x, r, lo);
  const int ii = lo[0] + di, jj = lo[1] + dj, kk = lo[2] + dk;
  const long long cell = (long long)ii + (long long)jj * xc + (long long)kk * yc * xc;
  int target = -1;
  double f[3] = {0.0, 0.0, 0.0};
  if (cell < a.C && cell >= 0) {
    const double wx = 1 - fabs(ii + 0.5 - r[0]);
    const double wy = 1 - fabs(jj + 0.5 - r[1]);
    const double wz = 1 - fabs(kk + 0.5 - r[2]);
    target = a.ibm_map[cell];
#pragma unroll
    for (int c = 0; c < 3; c++) f[c] = fn[c] * wx * wy * wz * a.ibm_inv_dx3;
  }
  spread_aggregated(act, target, f, a.force_x, a.force_y, a.force_z);
}

// FP64 node positions and forces; velocities interpolated from the FP32 state
// (times U) and forces spread as force / U in FP32.
__device__ __forceinline__ void ibm_thread32(const KernelArgs& a, const int t) {
  const int slot = t >> 3, sub = t & 7;
  const bool active = slot < a.N;
  const int nd = active ? __ldg(a.ibm_order + slot) : 0;
  const int xc = a.ibm_xc, yc = a.ibm_yc;
  const double U = a.uref;
  double x[3] = {0.0, 0.0, 0.0}, r[3] = {0.0, 0.0, 0.0};
  int lo[3] = {0, 0, 0};
  if (active) {
#pragma unroll
    for (int c = 0; c < 3; c++) x[c] = a.node_x[3 * nd + c];
    stencil_origin(a, x, r, lo);
  }
  const int di = sub & 1, dj = (sub >> 1) & 1, dk = sub >> 2;
  double v[3] = {0.0, 0.0, 0.0};
  {
    const int ii = lo[0] + di, jj = lo[1] + dj, kk = lo[2] + dk;
    const long long cell = (long long)ii + (long long)jj * xc + (long long)kk * yc * xc;
    if (active && cell < a.C && cell >= 0) {
      const double wx = 1 - fabs(ii + 0.5 - r[0]);
      const double wy = 1 - fabs(jj + 0.5 - r[1]);
      const double wz = 1 - fabs(kk + 0.5 - r[2]);
      const f4 q = ldf_rw(a.state, a.ibm_map[cell]);
      v[0] = __dmul_rn((U * q.x) * wx * wy * wz, a.ibm_inv_dx3);
      v[1] = __dmul_rn((U * q.y) * wx * wy * wz, a.ibm_inv_dx3);
      v[2] = __dmul_rn((U * q.z) * wx * wy * wz, a.ibm_inv_dx3);
    }
  }
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1)
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] += __shfl_xor_sync(full, v[c], o);
  const unsigned act = __ballot_sync(full, active);
  if (!active) return;
  double fn[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    x[c] = fma(v[c], a.dt, a.node_x0[3 * nd + c]);
    fn[c] = -a.ibm_area_k * (x[c] - a.node_ref[3 * nd + c]);
  }
  if (sub == 0) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      a.node_x[3 * nd + c] = x[c];
      a.node_x0[3 * nd + c] = x[c];
      a.node_vel[3 * nd + c] = v[c];
      a.node_force[3 * nd + c] = fn[c];
    }
  }
  stencil_origin(a, x, r, lo);
  const int ii = lo[0] + di, jj = lo[1] + dj, kk = lo[2] + dk;
  const long long cell = (long long)ii + (long long)jj * xc + (long long)kk * yc * xc;
  int target = -1;
  float f[3] = {0.f, 0.f, 0.f};
  if (cell < a.C && cell >= 0) {
    const double wgt = (1 - fabs(ii + 0.5 - r[0])) * (1 - fabs(jj + 0.5 - r[1])) *
                       (1 - fabs(kk + 0.5 - r[2])) * a.ibm_inv_dx3 / U;
    target = a.ibm_map[cell];
#pragma unroll
    for (int c = 0; c < 3; c++) f[c] = (float)(fn[c] * wgt);
  }
  spread_aggregated(act, target, f, a.fforce_x, a.fforce_y, a.fforce_z);
}

}  // namespace
}  // namespace plfbs
