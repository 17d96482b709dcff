// sm_100a kernels of the FP32 deviation form (PLFBS_FP32_DEVIATION).
//
// Same step structure as kernels.cu (gradient -> flux -> gather+RK per stage,
// IBM once per step), with state, gradients, fluxes, geometry and weights in
// FP32 and the variables shifted and scaled so that FP32 keeps the precision
// the residual needs:
//   state  (u/U, v/U, w/U, rho - rho0)
//   t0,t1  the RK accumulators in the same units (momentum / U, rho - rho0)
//   flux   (momentum flux / U, mass flux) with the constant rho0/3 n A part of
//          the momentum flux removed: it telescopes to zero over every closed
//          cell (sum_f n_f A_f = 0), so only deviations are carried.
// The equilibrium at a lattice node is split the same way:
//   feq = w rho0 + w [drho + rho U phi],
//   phi = 3 e.u' + 4.5 U (e.u')^2 / gamma - 1.5 U |u'|^2 / gamma,  u' = u/U,
// and the w rho0 part, whose moments are (rho0, 0, rho0/3 I), is left out of
// every sum. The residual norms are reduced in FP64, the Lagrangian node
// positions and forces stay FP64 (forces are spread as FP32 / U).
#include <cuda_runtime.h>

#include <cstdint>

#include "flux_core32.cuh"
#include "ibm_core.cuh"
#include "plfbs_internal.hpp"
#include "residual_core.cuh"

namespace plfbs {
namespace {

// Whether the context has converged or diverged. One thread per block reads
// the flag; every thread of the block must call this (it synchronises).
__device__ __forceinline__ bool halted(const KernelArgs& a) {
  __shared__ int h;
  if (threadIdx.x == 0) h = *(volatile const int*)&a.stats->halt;
  __syncthreads();
  return h != 0;
}

// Gradient layout: 3 x float4 per cell: (rx ry rz ux)(uy uz vx vy)(vz wx wy wz).
// Stencil slots as in k_gradient: neighbour ids first, then the slots.
template <bool CW>
__device__ __forceinline__ void gradient_slot32(const KernelArgs& a, long long s, int j,
                                                const f4& qi, float g[12], const float* wrow) {
  f4 qj;
  if (j < a.C) {
    qj = ldf(a.state, j);
  } else {
    const int b = j - a.C;
    const f4 tgt = ldf(a.bc1, b);
    const int types = (int)__ldg(reinterpret_cast<const float*>(a.bc3) + 4LL * b + 3);
    qj = ghost_state32(qi, tgt, types);
    stf(a.state, j, qj);
  }
  // CW: the cell's weight set from the compact table (wrow = its slot's triple)
  const float w[3] = {CW ? __ldg(wrow) : __ldg(static_cast<const float*>(a.st_wx) + s),
                      CW ? __ldg(wrow + 1) : __ldg(static_cast<const float*>(a.st_wy) + s),
                      CW ? __ldg(wrow + 2) : __ldg(static_cast<const float*>(a.st_wz) + s)};
  const float d[4] = {qj.w - qi.w, qj.x - qi.x, qj.y - qi.y, qj.z - qi.z};
#pragma unroll
  for (int f = 0; f < 4; f++)
#pragma unroll
    for (int c = 0; c < 3; c++) g[3 * f + c] = fmaf(w[c], d[f], g[3 * f + c]);
}

template <bool CW>
__global__ void __launch_bounds__(kBlock) k_gradient32(const KernelArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (halted(a)) return;
  if (i >= a.C) return;
  const f4 qi = ldf(a.state, i);
  const float* wset =
      CW ? static_cast<const float*>(a.wtab) + (size_t)__ldg(a.cell_wset + i) * a.K * 3 : nullptr;
  float g[12];
#pragma unroll
  for (int k = 0; k < 12; k++) g[k] = 0.0f;
  constexpr int kUnroll = 8;
  if (a.K <= kUnroll) {
    int jj[kUnroll];
#pragma unroll
    for (int k = 0; k < kUnroll; k++) jj[k] = k < a.K ? __ldg(a.st_nbr + (long long)k * a.C + i) : -1;
#pragma unroll
    for (int k = 0; k < kUnroll; k++)
      if (jj[k] >= 0)
        gradient_slot32<CW>(a, (long long)k * a.C + i, jj[k], qi, g, CW ? wset + 3 * k : nullptr);
  } else {
    for (int k = 0; k < a.K; k++) {
      const long long s = (long long)k * a.C + i;
      const int j = __ldg(a.st_nbr + s);
      if (j < 0) break;
      gradient_slot32<CW>(a, s, j, qi, g, CW ? wset + 3 * k : nullptr);
    }
  }
  stf(a.grad, 3LL * i + 0, f4{g[0], g[1], g[2], g[3]});
  stf(a.grad, 3LL * i + 1, f4{g[4], g[5], g[6], g[7]});
  stf(a.grad, 3LL * i + 2, f4{g[8], g[9], g[10], g[11]});
}

// Face flux in deviation form (see the file comment).
// CR: the face's records from the compact tables (rec = its index there).
template <bool CR>
__device__ __forceinline__ void flux_face32(const KernelArgs& a, const int f, const int2 ids,
                                            const int rec) {
  const f4 f0 = CR ? ldf(a.frec0, rec) : ldf(a.face0, f);
  const f4 f1 = CR ? ldf(a.frec1, rec) : ldf(a.face1, f);
  const f4 f2 = CR ? ldf(a.frec2, rec) : ldf(a.face2, f);
  const int o = ids.x, nb = ids.y;
  const float n[3] = {f0.x, f0.y, f0.z}, dt = f1.x;
  const float t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
  const f4 qo = ldf(a.state, o);
  float g1[12], g2[12], si[4], sn[4], sc[4];
  load_grad32(a.grad, o, g1);
  unsigned sides = CR ? (unsigned)__ldg(a.frec_sides + rec) : 0u;
  if (nb < a.C) {
    const f4 qn = ldf(a.state, nb);
    load_grad32(a.grad, nb, g2);
    if (CR && (sides >> kKindShift)) {
      const unsigned kind = sides >> kKindShift;
      const f4 x =
          kind == 1 ? axis_flux32<0>(a, dt, t1[0], t2[0], n[0], f0.w, f2.w, qo, qn, g1, g2)
          : kind == 2 ? axis_flux32<1>(a, dt, t1[1], t2[1], n[1], f0.w, f2.w, qo, qn, g1, g2)
                      : axis_flux32<2>(a, dt, t1[2], t2[2], n[2], f0.w, f2.w, qo, qn, g1, g2);
      stf(a.flux, f, x);
      return;
    }
    interior_sides32(t1, t2, qo, qn, g1, g2, si, sn, sc);
  } else {
    boundary_sides32(a, nb - a.C, t1, t2, qo, g1, g2, si, sn, sc);
  }
  if (!CR) sides = face_sides32(n[0], n[1], n[2], __fmul_rn(0.001f, dt));
  stf(a.flux, f, face_flux32(a, n, f0.w, f2.w, sides, dt, si, sn, sc, g1, g2));
}

// Persistent over the faces, next face's ids prefetched, int counters and the
// compact layout's block-uniform loop as in k_flux; six blocks per SM (85
// registers) measured fastest.
template <bool CR>
__global__ void __launch_bounds__(kFluxBlock, 6) k_flux32(const KernelArgs a) {
  if (halted(a)) return;
  const int2* face_ids = reinterpret_cast<const int2*>(a.face_ids);
  const int stride = gridDim.x * kFluxBlock;
  int f = blockIdx.x * kFluxBlock + threadIdx.x;
  if constexpr (CR) {
    const int tiles = (a.F + kFluxBlock - 1) / kFluxBlock;
    int2 ids = f < a.F ? __ldg(face_ids + f) : make_int2(0, 0);
    int rec = f < a.F ? __ldg(a.face_rec + f) : 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int fn = f + stride;
      const int2 next = fn < a.F ? __ldg(face_ids + fn) : make_int2(0, 0);
      const int next_rec = fn < a.F ? __ldg(a.face_rec + fn) : 0;
      if (f < a.F) flux_face32<CR>(a, f, ids, rec);
      f = fn;
      ids = next;
      rec = next_rec;
    }
  } else {
    if (f >= a.F) return;
    int2 ids = __ldg(face_ids + f);
    for (;;) {
      const int fn = f + stride;
      const int2 next = fn < a.F ? __ldg(face_ids + fn) : make_int2(0, 0);
      flux_face32<CR>(a, f, ids, 0);
      if (fn >= a.F) break;
      f = fn;
      ids = next;
    }
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Gather + body force + RK stage in deviation units; the last stage reduces
// the squared residuals in FP64 (momentum residuals are already divided by U,
// so inv_ref_mom is 1 / rho_ref here).
template <int RK, int K2MAX>
__global__ void __launch_bounds__(kBlock) k_update32(const KernelArgs a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (halted(a)) return;
  if (RK == 3 && a.red_order) i = i < a.C ? __ldg(a.red_order + i) : a.C;  // as k_update
  double sq[4] = {0.0, 0.0, 0.0, 0.0};
  bool bad = false;
  if (i < a.C) {
    // The RK accumulators a stage needs (as k_update), loaded first, with the
    // gather, so no store of the stage can come between them and the flux
    // loads.
    f4 t0{}, t1{};
    if (RK != 3) t0 = ldf_rw(a.t0, i);
    if (RK != 0) t1 = ldf_rw(a.t1, i);
    float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int e[K2MAX];
#pragma unroll
    for (int k = 0; k < K2MAX; k++) e[k] = (k < a.K2) ? __ldg(a.gather + (long long)k * a.C + i) : -1;
    f4 fl[K2MAX];
#pragma unroll
    for (int k = 0; k < K2MAX; k++)
      if (e[k] >= 0) fl[k] = ldf(a.flux, e[k] >> 1);
#pragma unroll
    for (int k = 0; k < K2MAX; k++) {
      if (e[k] < 0) continue;
      const float sg = (e[k] & 1) ? 1.0f : -1.0f;
      r[0] = fmaf(sg, fl[k].x, r[0]);
      r[1] = fmaf(sg, fl[k].y, r[1]);
      r[2] = fmaf(sg, fl[k].z, r[2]);
      r[3] = fmaf(sg, fl[k].w, r[3]);
    }
    const float iv = __ldg(static_cast<const float*>(a.inv_volume) + i);
    const float pgU = __fmul_rn((float)a.pressure_gradient, a.inv_uref_f);
    float fc[3] = {pgU, 0.0f, 0.0f};
    if (a.fforce_x) {
      fc[0] = a.fforce_x[i];
      fc[1] = a.fforce_y[i];
      fc[2] = a.fforce_z[i];
    }
    const float R[4] = {fmaf(r[0], iv, fc[0]), fmaf(r[1], iv, fc[1]), fmaf(r[2], iv, fc[2]),
                        r[3] * iv};
    if (a.res_debug) stf(a.res_debug, i, f4{R[0], R[1], R[2], R[3]});
    f4 q, acc;
    rk_stage32<RK>((float)a.dt, a.rho0f, t0, t1, R, q, acc);
    if (RK == 3) {
      sq[0] = (double)R[3] * R[3];
      sq[1] = (double)R[0] * R[0];
      sq[2] = (double)R[1] * R[1];
      sq[3] = (double)R[2] * R[2];
      bad = !(__fadd_rn(a.rho0f, acc.w) <= 1000.0f);
    }
    stf(RK == 3 ? a.t0 : a.t1, i, acc);
    stf(a.state, i, q);
    if (RK == 3 && a.fforce_x) {  // after every load of the stage (see k_update)
      a.fforce_x[i] = pgU;
      a.fforce_y[i] = 0.0f;
      a.fforce_z[i] = 0.0f;
    }
  }
  if (RK != 3) return;

  // Per-block squared-residual sums (warp shuffle, then the block's warps in
  // order); k_finish32 reduces them.
  __shared__ double red[kBlock / 32][4];
  __shared__ int any_bad;
  if (threadIdx.x == 0) any_bad = 0;
  __syncthreads();
  if (bad) atomicOr(&any_bad, 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const double v = warp_sum(sq[c]);
    if (lane == 0) red[warp][c] = v;
  }
  __syncthreads();
  if (a.red_order) {  // per warp of cells; k_finish adds them tile by tile
    const int w = threadIdx.x / 4, c = threadIdx.x & 3;
    const long long at = (long long)blockIdx.x * (kBlock / 32) + w;
    if (w < kBlock / 32 && 32 * at < a.C) a.partial[4 * at + c] = red[w][c];
  } else if (threadIdx.x < 4) {
    double v = 0.0;
    for (int w = 0; w < kBlock / 32; w++) v += red[w][threadIdx.x];
    a.partial[4LL * blockIdx.x + threadIdx.x] = v;
  }
  if (threadIdx.x == 0 && any_bad) a.stats->diverged = 1;
}

// One block after the last stage: sums the per-block partials in a fixed
// order, forms the rms norms of l2_norm_rms_moukallad (residuals.cpp:95-113)
// and max_error (:139-147), records the step and tests convergence
// (Solver_gpu.cu:870); a converged or diverged context halts.
__global__ void __launch_bounds__(kFinishBlock) k_finish32(const KernelArgs a) {
  if (halted(a)) return;
  __shared__ double red[kFinishBlock / 32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (a.red_order) tile_sums(a, v);
#pragma unroll 4
  for (int b = threadIdx.x; b < (a.red_order ? 0 : a.nblk_update); b += kFinishBlock) {
    const double2 p0 = __ldg(reinterpret_cast<const double2*>(a.partial + 4LL * b));
    const double2 p1 = __ldg(reinterpret_cast<const double2*>(a.partial + 4LL * b) + 1);
    v[0] += p0.x;
    v[1] += p0.y;
    v[2] += p1.x;
    v[3] += p1.y;
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const double w = warp_sum(v[c]);
    if (lane == 0) red[warp][c] = w;
  }
  __syncthreads();
  if (warp > 0) return;
  double rms = 0.0;  // a lane per component
  if (lane < 4) {
    double tot = 0.0;
    for (int w = 0; w < (a.red_order ? kMaxTiles / 32 : kFinishBlock / 32); w++) tot += red[w][lane];
    rms = sqrt(tot / (double)a.C) * (lane == 0 ? a.inv_ref_rho : a.inv_ref_mom);
  }
  const double rho_rms = __shfl_sync(0xffffffffu, rms, 0), u_rms = __shfl_sync(0xffffffffu, rms, 1),
               v_rms = __shfl_sync(0xffffffffu, rms, 2), w_rms = __shfl_sync(0xffffffffu, rms, 3);
  if (lane == 0) {
    DevStats* st = a.stats;
    const double me = fmax(fmax(w_rms, u_rms), v_rms);  // residuals::max_error
    const long long t = st->steps;
    double* h = st->history[t % kHistoryCap];
    h[0] = (double)t;
    h[1] = me;
    h[2] = rho_rms;
    h[3] = u_rms;
    h[4] = v_rms;
    h[5] = w_rms;
    for (int c = 0; c < 6; c++) st->last[c] = h[c];
    st->steps = t + 1;
    if (!(me == me) || !(rho_rms == rho_rms)) st->diverged = 1;
    if (me < a.tolerance) {
      st->converged = 1;
      st->converged_step = t;
    }
    if (st->converged || st->diverged) st->halt = 1;
  }
}

// As k_seed; the conserved accumulators in deviation units are
// (rho u / U, rho v / U, rho w / U, rho - rho0).
template <bool CONSERVED>
__global__ void k_seed32(const KernelArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.C) return;
  f4 q = ldf(a.state, i);
  if (CONSERVED) {
    const float rho = a.rho0f + q.w;
    q = f4{rho * q.x, rho * q.y, rho * q.z, q.w};
  }
  stf(a.t0, i, q);
}

__global__ void __launch_bounds__(kIbmBlock) k_ibm32(const KernelArgs a) {
  if (halted(a)) return;
  ibm_thread32(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// Branch bits of the compact layout's unique records.
__global__ void k_record_sides32(const void* frec0, const void* frec1, const void* frec2, int n,
                                 int32_t* out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const f4 f0 = ldf(frec0, r), f1 = ldf(frec1, r);
    const unsigned sides = face_sides32(f0.x, f0.y, f0.z, __fmul_rn(0.001f, f1.x));
    out[r] = (int32_t)(sides | face_kind32(f0, f1, ldf(frec2, r), sides) << kKindShift);
  }
}

inline int blocks_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

template <int RK>
void launch_update32_rk(const KernelArgs& a, cudaStream_t s) {
  const int nb = blocks_for(a.C, kBlock);
  if (a.K2 <= 4)
    k_update32<RK, 4><<<nb, kBlock, 0, s>>>(a);
  else if (a.K2 <= 6)
    k_update32<RK, 6><<<nb, kBlock, 0, s>>>(a);
  else if (a.K2 <= 8)
    k_update32<RK, 8><<<nb, kBlock, 0, s>>>(a);
  else
    k_update32<RK, 16><<<nb, kBlock, 0, s>>>(a);
}

}  // namespace

void launch_record_sides32(const void* frec0, const void* frec1, const void* frec2, int n,
                           int32_t* out, cudaStream_t s) {
  k_record_sides32<<<blocks_for(n, kBlock), kBlock, 0, s>>>(frec0, frec1, frec2, n, out);
}

void launch_gradient32(const KernelArgs& a, cudaStream_t s) {
  if (a.compact && a.wtab)
    k_gradient32<true><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
  else
    k_gradient32<false><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
}
void launch_flux32(const KernelArgs& a, cudaStream_t s) {
  static std::atomic<int> resident[kMaxDevices], cr_resident[kMaxDevices];
  if (a.compact && a.face_rec)
    k_flux32<true><<<persistent_blocks(k_flux32<true>, kFluxBlock, a.F, cr_resident), kFluxBlock,
                     0, s>>>(a);
  else
    k_flux32<false><<<persistent_blocks(k_flux32<false>, kFluxBlock, a.F, resident), kFluxBlock,
                      0, s>>>(a);
}
void launch_update32(const KernelArgs& a, int rk, cudaStream_t s, bool finish) {
  switch (rk) {
    case 0: launch_update32_rk<0>(a, s); break;
    case 1: launch_update32_rk<1>(a, s); break;
    case 2: launch_update32_rk<2>(a, s); break;
    default:
      launch_update32_rk<3>(a, s);
      if (finish) k_finish32<<<1, kFinishBlock, 0, s>>>(a);
      break;
  }
}
void launch_finish32(const KernelArgs& a, cudaStream_t s) {
  k_finish32<<<1, kFinishBlock, 0, s>>>(a);
}
void launch_seed32(const KernelArgs& a, bool conserved, cudaStream_t s) {
  if (conserved)
    k_seed32<true><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
  else
    k_seed32<false><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
}
void launch_ibm32(const KernelArgs& a, cudaStream_t s) {
  if (a.N > 0) k_ibm32<<<blocks_for(8LL * a.N, kIbmBlock), kIbmBlock, 0, s>>>(a);
}

}  // namespace plfbs
