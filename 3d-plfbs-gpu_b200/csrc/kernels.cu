// sm_100a kernels of the LBFS explicit time step (FP64 path).
//
// One RK stage is three kernels, and a time step is the IBM kernel plus four
// stages, all captured in one CUDA graph by capi.cpp (a mesh small enough
// marches in one cooperative kernel instead, march.cu, and uses these stage by
// stage only):
//
//   gradient  (thread per cell)  ghost states inline + least-squares gradient
//                                 [get_interior_gradients, update_unstructured_bcs]
//   flux      (thread per face)  D3Q15 reconstruction + interface equilibrium
//                                 + relaxed moment flux, written per face
//                                 [calc_face_flux, get_bc_gradients]
//   update    (thread per cell)  face->cell gather (no atomics) + body force +
//                                 RK stage; last stage also reduces residuals
//                                 and tests convergence on the device
//                                 [add, time_integration, square/total<256>,
//                                  l2_norm_rms_moukallad]
//   ibm       (8 threads/node)   interpolation, advection, spring force and
//                                 spreading with FP64 atomics
//
// All of them are bandwidth kernels (no dense contraction: tensor cores do not
// apply). Memory per cell is laid out for coalesced 32-byte accesses.
#include <cuda_runtime.h>

#include <cstdint>

#include "flux_core.cuh"
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

// ---------------------------------------------------------------------------
// gradient: grad_i = sum_e G_e (q_e - q_i), G_e = LHS_i^-1 RHS_e precombined.
// Gradient layout: 3 x d4 per cell = (rx, ry, rz, ux), (uy, uz, vx, vy),
// (vz, wx, wy, wz).
// ---------------------------------------------------------------------------
// One thread per cell. The neighbour ids of up to kStencilUnroll slots are
// loaded first, then every slot's weights and neighbour state, so a cell waits
// for two rounds of loads rather than two per slot; wider stencils fall back
// to walking the slots.
template <bool GHOSTS, int FL, bool CW>
__device__ __forceinline__ void gradient_slot(const KernelArgs& a, int i, long long s, int j,
                                              const d4& qi, double g[12], const double* wrow) {
  d4 qj;
  if (!GHOSTS || j < a.C) {
    qj = ld4(a.state, j);
  } else {
    const int b = j - a.C;
    const d4 tgt = ld4(a.bc1, b);
    const int types = (int)__ldg(reinterpret_cast<const double*>(a.bc3) + 4LL * b + 3);
    qj = ghost_state<FL>(qi, tgt, types);
    st4(a.state, j, qj);  // the ghost's only reader in this kernel is its owner
  }
  // CW: the cell's weight set from the compact table (wrow = its slot's triple)
  const double w[3] = {CW ? __ldg(wrow) : __ldg(static_cast<const double*>(a.st_wx) + s),
                       CW ? __ldg(wrow + 1) : __ldg(static_cast<const double*>(a.st_wy) + s),
                       CW ? __ldg(wrow + 2) : __ldg(static_cast<const double*>(a.st_wz) + s)};
  const double d[4] = {qj.w - qi.w, qj.x - qi.x, qj.y - qi.y, qj.z - qi.z};
#pragma unroll
  for (int f = 0; f < 4; f++)
#pragma unroll
    for (int c = 0; c < 3; c++) g[3 * f + c] = fma(w[c], d[f], g[3 * f + c]);
}

constexpr int kStencilUnroll = 8;

template <int FL, bool CW>
__global__ void __launch_bounds__(kBlock) k_gradient(const KernelArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (halted(a)) return;
  if (i >= a.C) return;
  const d4 qi = ld4(a.state, i);
  const double* wset =
      CW ? static_cast<const double*>(a.wtab) + (size_t)__ldg(a.cell_wset + i) * a.K * 3 : nullptr;
  double g[12];
#pragma unroll
  for (int k = 0; k < 12; k++) g[k] = 0.0;
  if (a.K <= kStencilUnroll) {
    int jj[kStencilUnroll];
#pragma unroll
    for (int k = 0; k < kStencilUnroll; k++)
      jj[k] = k < a.K ? __ldg(a.st_nbr + (long long)k * a.C + i) : -1;
#pragma unroll
    for (int k = 0; k < kStencilUnroll; k++)
      if (jj[k] >= 0)
        gradient_slot<true, FL, CW>(a, i, (long long)k * a.C + i, jj[k], qi, g,
                                    CW ? wset + 3 * k : nullptr);
  } else {
    for (int k = 0; k < a.K; k++) {
      const long long s = (long long)k * a.C + i;
      const int j = __ldg(a.st_nbr + s);
      if (j < 0) break;
      gradient_slot<true, FL, CW>(a, i, s, j, qi, g, CW ? wset + 3 * k : nullptr);
    }
  }
  st4(a.grad, 3LL * i + 0, d4{g[0], g[1], g[2], g[3]});
  st4(a.grad, 3LL * i + 1, d4{g[4], g[5], g[6], g[7]});
  st4(a.grad, 3LL * i + 2, d4{g[8], g[9], g[10], g[11]});
}

// ---------------------------------------------------------------------------
// flux
// ---------------------------------------------------------------------------
__device__ __forceinline__ int2 face_ids(const KernelArgs& a, long long f) {
  return __ldg(reinterpret_cast<const int2*>(a.face_ids) + f);
}

// CR: the face's records from the compact tables (rec = its index there).
template <int FL, bool CR>
__device__ __forceinline__ void flux_face(const KernelArgs& a, const int f, const int2 ids,
                                          const int rec) {
  const int r = CR ? rec : f;
  const d4 f0 = ld4(CR ? a.frec0 : a.face0, r), f1 = ld4(CR ? a.frec1 : a.face1, r),
           f2 = ld4(CR ? a.frec2 : a.face2, r);
  const int o = ids.x, nb = ids.y;
  const double dt = f1.x;
  // the branch decisions: per record with the compact layout (FP64 compact
  // layouts always carry them)
  unsigned sides = CR ? (unsigned)__ldg(a.frec_sides + r) : 0u;
  const d4 qo = ld4(a.state, o);
  double g1[12], g2[12], si[4], sn[4], sc[4];
  load_grad(a.grad, o, g1);
  const double t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
  if (nb < a.C) {
    const d4 qn = ld4(a.state, nb);
    load_grad(a.grad, nb, g2);
    if (CR && (sides >> kKindShift)) {
      const double2 w = __ldg(reinterpret_cast<const double2*>(a.frec_relax) + r);
      const unsigned kind = sides >> kKindShift;
      const d4 x =
          kind == 1 ? axis_flux<FL, 0>(a, dt, t1[0], t2[0], f0.x, f0.w, w.x, w.y, qo, qn, g1, g2)
          : kind == 2 ? axis_flux<FL, 1>(a, dt, t1[1], t2[1], f0.y, f0.w, w.x, w.y, qo, qn, g1, g2)
                      : axis_flux<FL, 2>(a, dt, t1[2], t2[2], f0.z, f0.w, w.x, w.y, qo, qn, g1, g2);
      st4(a.flux, f, x);
      return;
    }
    interior_sides(t1, t2, qo, qn, g1, g2, si, sn, sc);
  } else {
    boundary_sides<FL>(a, nb - a.C, t1, t2, qo, g1, g2, si, sn, sc);
  }
  const double n[3] = {f0.x, f0.y, f0.z};
  if (!CR) sides = face_sides<FL>(n, dt);
  st4(a.flux, f, face_flux<FL, CR>(a, r, sides, dt, si, sn, sc, g1, g2));
}

// Persistent over the faces [f_begin, f_end) (grid stride): the
// owner/neighbour ids of a thread's next face are loaded before its current
// face is computed, so the next face's cell gathers do not wait behind a load
// of its face record. Four blocks per SM (128 registers) measured faster than
// three without spills (73 vs 75 us) and than five or six with more spills
// (102, 191 us): latency hiding wins until the spills take over. A face index
// fits in 31 bits (the gather lists hold it doubled), so the loop counts in
// int: with 64-bit counters the spills cost 421 us against 387 on the compact
// 256 x 128 x 128 mesh. On the compact layout the loop also stays uniform over
// the block, with the ragged last tile predicated (387 -> 371 us);
// per-item records, whose registers differ, measured 2-4 % faster with each
// thread leaving by itself (147 vs 153 us on 1.57 M tetrahedra).
template <int FL, bool CR>
__global__ void __launch_bounds__(kFluxBlock, 4) k_flux(const KernelArgs a, int f_begin,
                                                        int f_end) {
  if (halted(a)) return;
  const int stride = gridDim.x * kFluxBlock;
  int f = f_begin + blockIdx.x * kFluxBlock + threadIdx.x;
  if constexpr (CR) {
    const int tiles = (f_end - f_begin + kFluxBlock - 1) / kFluxBlock;
    int2 ids = f < f_end ? face_ids(a, f) : make_int2(0, 0);
    int rec = f < f_end ? __ldg(a.face_rec + f) : 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int fn = f + stride;
      const int2 next = fn < f_end ? face_ids(a, fn) : make_int2(0, 0);
      const int next_rec = fn < f_end ? __ldg(a.face_rec + fn) : 0;
      if (f < f_end) flux_face<FL, CR>(a, f, ids, rec);
      f = fn;
      ids = next;
      rec = next_rec;
    }
  } else {
    if (f >= f_end) return;
    int2 ids = face_ids(a, f);
    for (;;) {
      const int fn = f + stride;
      const int2 next = fn < f_end ? face_ids(a, fn) : make_int2(0, 0);
      flux_face<FL, CR>(a, f, ids, 0);
      if (fn >= f_end) break;
      f = fn;
      ids = next;
    }
  }
}

// ---------------------------------------------------------------------------
// flux, TMA-staged (internal faces): a producer warp gathers each tile's cell
// rows into shared memory with tile::gather4 bulk tensor copies while four
// consumer warps compute the previous tile. The consumers never wait on a
// global gather; the arithmetic per face is face_flux's.
// ---------------------------------------------------------------------------
constexpr int kTmaFaces = 128;  // faces per tile, one per consumer thread
constexpr int kTmaStages = 2;
constexpr int kTmaThreads = kTmaFaces + 32;
// stage layout (bytes): owner state rows, neighbour state rows, owner
// gradient rows, neighbour gradient rows
constexpr int kTmaSo = 0, kTmaSn = kTmaFaces * 32, kTmaGo = 2 * kTmaFaces * 32,
              kTmaGn = kTmaGo + kTmaFaces * 96, kTmaStageBytes = kTmaGn + kTmaFaces * 96;
// + room to align the stages to 128 bytes by hand (bulk tensor copies need it)
constexpr int kTmaSmem = kTmaStages * kTmaStageBytes + 2 * kTmaStages * 8 + 128;
constexpr int kSpinLimit = 1 << 22;  // try_wait rounds before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}
// Waits for the phase of the given parity; false after kSpinLimit tries.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) {
  for (int i = 0; i < kSpinLimit; i++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// Rows r[0..3] (column 0) of a 2D tensor map into consecutive boxes at dst.
__device__ __forceinline__ void gather4(void* dst, const CUtensorMap* map, const int r[4],
                                        uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
      "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void report_fault(const KernelArgs& a) {
  atomicExch(&a.stats->fault, 1);
  atomicExch(&a.stats->halt, 1);
}

__global__ void __launch_bounds__(kTmaThreads, 3)
    k_flux_tma(const KernelArgs a, const __grid_constant__ FluxMaps maps) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (halted(a)) return;
  unsigned char* smem = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kTmaStages * kTmaStageBytes);
  uint64_t* empty = full + kTmaStages;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kTmaStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kTmaFaces / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int ntiles = (a.Fi + kTmaFaces - 1) / kTmaFaces;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == kTmaFaces / 32) {
    // producer: four faces per lane, one gather4 per row kind
    int k = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, k++) {
      const int s = k % kTmaStages;
      if (k >= kTmaStages && !mbar_wait(&empty[s], (k / kTmaStages - 1) & 1)) {
        report_fault(a);
        return;
      }
      int own[4], nbr[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int f = t * kTmaFaces + 4 * lane + j;
        const int2 id = f < a.Fi ? face_ids(a, f) : make_int2(0, 0);  // past the end: cell 0
        own[j] = id.x;
        nbr[j] = id.y;
      }
      if (lane == 0) mbar_expect_tx(&full[s], kTmaStageBytes);
      __syncwarp();
      unsigned char* st = smem + s * kTmaStageBytes;
      gather4(st + kTmaSo + 128 * lane, &maps.state, own, &full[s]);
      gather4(st + kTmaSn + 128 * lane, &maps.state, nbr, &full[s]);
      gather4(st + kTmaGo + 384 * lane, &maps.grad, own, &full[s]);
      gather4(st + kTmaGn + 384 * lane, &maps.grad, nbr, &full[s]);
    }
    return;
  }
  // consumers: one face per thread per tile
  const int c = threadIdx.x;
  int k = 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, k++) {
    const int s = k % kTmaStages;
    const int f = t * kTmaFaces + c;
    const bool valid = f < a.Fi;
    d4 f0{}, f1{}, f2{};
    if (valid) {  // face records: contiguous, issued before the wait
      f0 = ld4(a.face0, f);
      f1 = ld4(a.face1, f);
      f2 = ld4(a.face2, f);
    }
    if (!mbar_wait(&full[s], (k / kTmaStages) & 1)) {
      report_fault(a);
      mbar_wait(&full[s], (k / kTmaStages) & 1);  // let copies in flight land
      return;
    }
    const unsigned char* st = smem + s * kTmaStageBytes;
    const double* so = reinterpret_cast<const double*>(st + kTmaSo) + 4 * c;
    const double* sn_ = reinterpret_cast<const double*>(st + kTmaSn) + 4 * c;
    const double* go = reinterpret_cast<const double*>(st + kTmaGo) + 12 * c;
    const double* gn = reinterpret_cast<const double*>(st + kTmaGn) + 12 * c;
    // state rows are (u, v, w, rho), read before the stage is handed back
    const d4 qo{so[0], so[1], so[2], so[3]}, qn{sn_[0], sn_[1], sn_[2], sn_[3]};
    double g1[12], g2[12];
#pragma unroll
    for (int i = 0; i < 12; i++) {
      g1[i] = go[i];
      g2[i] = gn[i];
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (!valid) continue;
    const double n[3] = {f0.x, f0.y, f0.z};
    const double dt = f1.x;
    const double t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
    double si[4], sn[4], sc[4];
    interior_sides(t1, t2, qo, qn, g1, g2, si, sn, sc);
    st4(a.flux, f, face_flux<0, false>(a, f, face_sides<0>(n, dt), dt, si, sn, sc, g1, g2));
  }
}

// ---------------------------------------------------------------------------
// update: gather + body force + RK stage (time_integration, LBFS.cu:1457-1521)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// K2MAX: face slots the launch is specialised for (0 = any count, looped).
template <int RK, int K2MAX>
__global__ void __launch_bounds__(kBlock) k_update(const KernelArgs a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (halted(a)) return;  // uniform across the launch
  // a context that marches sums its residuals along its tiles
  if (RK == 3 && a.red_order) i = i < a.C ? __ldg(a.red_order + i) : a.C;
  double sq[4] = {0.0, 0.0, 0.0, 0.0};
  bool bad = false;
  if (i < a.C) {
    // The RK accumulators are loaded first, with the gather, so no store of
    // the stage can come between them and the flux loads. A stage moves only
    // those it needs (rk_stage): the step's start t0 in stages 0-2, the
    // accumulator t1 read in 1-3 and written in 0-2, the finished one to t0.
    d4 t0{}, t1{};
    if (RK != 3) t0 = ld4rw(a.t0, i);
    if (RK != 0) t1 = ld4rw(a.t1, i);
    double r[4] = {0.0, 0.0, 0.0, 0.0};
    if (K2MAX > 0) {
      int e[K2MAX > 0 ? K2MAX : 1];
#pragma unroll
      for (int k = 0; k < K2MAX; k++) e[k] = (k < a.K2) ? __ldg(a.gather + (long long)k * a.C + i) : -1;
      d4 fl[K2MAX > 0 ? K2MAX : 1];
#pragma unroll
      for (int k = 0; k < K2MAX; k++)
        if (e[k] >= 0) fl[k] = ld4(a.flux, e[k] >> 1);
#pragma unroll
      for (int k = 0; k < K2MAX; k++) {
        if (e[k] < 0) continue;
        const double sg = (e[k] & 1) ? 1.0 : -1.0;
        r[0] = fma(sg, fl[k].x, r[0]);
        r[1] = fma(sg, fl[k].y, r[1]);
        r[2] = fma(sg, fl[k].z, r[2]);
        r[3] = fma(sg, fl[k].w, r[3]);
      }
    } else {
      for (int k = 0; k < a.K2; k++) {
        const int e = __ldg(a.gather + (long long)k * a.C + i);
        if (e < 0) break;
        const d4 fl = ld4(a.flux, e >> 1);
        const double sg = (e & 1) ? 1.0 : -1.0;
        r[0] = fma(sg, fl.x, r[0]);
        r[1] = fma(sg, fl.y, r[1]);
        r[2] = fma(sg, fl.z, r[2]);
        r[3] = fma(sg, fl.w, r[3]);
      }
    }
    const double iv = __ldg(static_cast<const double*>(a.inv_volume) + i);
    double fc[3] = {a.pressure_gradient, 0.0, 0.0};
    if (a.force_x) {
      fc[0] = a.force_x[i];
      fc[1] = a.force_y[i];
      fc[2] = a.force_z[i];
    }
    const double R[4] = {fma(r[0], iv, fc[0]), fma(r[1], iv, fc[1]), fma(r[2], iv, fc[2]),
                         r[3] * iv};  // u, v, w, rho
    if (a.res_debug) st4(a.res_debug, i, d4{R[0], R[1], R[2], R[3]});
    d4 q, acc;
    rk_stage<RK>(a.dt, t0, t1, R, q, acc);
    if (RK == 3) {
      sq[0] = R[3] * R[3];
      sq[1] = R[0] * R[0];
      sq[2] = R[1] * R[1];
      sq[3] = R[2] * R[2];
      bad = !(acc.w <= 1000.0);  // the CPU solver's divergence test, Solver.cpp:448-493
    }
    st4(RK == 3 ? a.t0 : a.t1, i, acc);
    st4(a.state, i, q);
    // The last reader of this step's force resets it for the IBM. The stores
    // come after every load of the stage: placed before the t0/t1 loads they
    // would hold those loads back (the pointers may alias).
    if (RK == 3 && a.force_x) {
      a.force_x[i] = a.pressure_gradient;
      a.force_y[i] = 0.0;
      a.force_z[i] = 0.0;
    }
  }
  if (RK != 3) return;

  // Per-block squared-residual sums (warp shuffle, then the block's warps in
  // order); k_finish reduces them.
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
__global__ void __launch_bounds__(kFinishBlock) k_finish(const KernelArgs a) {
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

// Seeds the RK accumulator from the state (Solver_gpu.cu:664): t0 = q (t1 is
// written by the first stage before it is read). The reference seeds the velocity state although the stages treat t0/t1 as
// (rho u, rho v, rho w, rho); with conserved = true (warm starts, no reference
// counterpart) the accumulators get the conserved variables instead.
template <bool CONSERVED>
__global__ void k_seed(const KernelArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.C) return;
  d4 q = ld4(a.state, i);
  if (CONSERVED) q = d4{q.w * q.x, q.w * q.y, q.w * q.z, q.w};
  st4(a.t0, i, q);
}

// The immersed body (ibm_core.cuh), once per time step before the RK stages.
__global__ void __launch_bounds__(kIbmBlock) k_ibm(const KernelArgs a) {
  if (halted(a)) return;
  ibm_thread(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Wall forces of post_processing::cylinder_post_processing
// (post_processing.cpp:50-173) over the listed boundary faces (internal bc
// indices), from the current state and gradients (the reference calls it
// after update_unstructured_bcs and Get_LS_Gradients on the host, so the
// ghost gradients follow the host rules of gradients.cpp:441-463 and 592-645:
// Dirichlet velocity 2 (u_b - u_o) / |d| times the face normal, Neumann the
// owner's gradient times (1 - n)). Per face: p = rho_o gamma / 3,
//   drag += ((p - nu gamma du/dx) n_x - nu gamma du/dy n_y) A
//   lift += (nu gamma dv/dx n_x - (p - nu gamma dv/dy) n_y) A.
// One block; the partial sums are added in a fixed order. out[2] = {drag, lift}.
// ---------------------------------------------------------------------------
constexpr int kWallBlock = 1024;

__global__ void __launch_bounds__(kWallBlock) k_wall_forces(const KernelArgs a, const int* walls,
                                                            int n, int fp32, double visc_g,
                                                            double gamma, double* out) {
  __shared__ double red[kWallBlock / 32][2];
  double dr = 0.0, li = 0.0;
  const long long Fi = (long long)a.F - a.B;  // boundary face of bc b: Fi + b
  for (int k = threadIdx.x; k < n; k += kWallBlock) {
    const int b = walls[k];
    const long long f = Fi + b;
    const int o = a.face_ids[2 * f];
    double nx, ny, area, rho, uo, vo, ub, vb, dmag, gux, guy, gvx, gvy;
    int types;
    if (fp32) {  // deviation units: velocity / U, rho - rho0
      const float4 f0 = reinterpret_cast<const float4*>(a.face0)[f];
      const float4 q = reinterpret_cast<const float4*>(a.state)[o];
      const float4 bv = reinterpret_cast<const float4*>(a.bc0)[b];
      const float4 dd = reinterpret_cast<const float4*>(a.bc2)[b];
      const float4 nm = reinterpret_cast<const float4*>(a.bc3)[b];
      const float4 g0 = reinterpret_cast<const float4*>(a.grad)[3LL * o];
      const float4 g1 = reinterpret_cast<const float4*>(a.grad)[3LL * o + 1];
      const double U = a.uref;
      nx = f0.x; ny = f0.y; area = f0.w;
      rho = a.rho0 + q.w;
      uo = U * q.x; vo = U * q.y; ub = U * bv.x; vb = U * bv.y;
      dmag = dd.w;
      types = (int)nm.w;
      gux = U * g0.w; guy = U * g1.x; gvx = U * g1.z; gvy = U * g1.w;
    } else {
      const d4 f0 = ld4(a.face0, f), q = ld4(a.state, o), bv = ld4(a.bc0, b), dd = ld4(a.bc2, b),
               nm = ld4(a.bc3, b), g0 = ld4(a.grad, 3LL * o), g1 = ld4(a.grad, 3LL * o + 1);
      nx = f0.x; ny = f0.y; area = f0.w;
      rho = q.w;
      uo = q.x; vo = q.y; ub = bv.x; vb = bv.y;
      dmag = dd.w;
      types = (int)nm.w;
      gux = g0.w; guy = g1.x; gvx = g1.z; gvy = g1.w;
    }
    double ux, uy, vx, vy;
    if ((types >> 8) == 1) {  // Dirichlet velocity: get_ghost_grads
      const double du = 2 * (ub - uo), dv = 2 * (vb - vo);
      ux = du / dmag * nx;
      uy = du / dmag * ny;
      vx = dv / dmag * nx;
      vy = dv / dmag * ny;
    } else {  // Neumann velocity (the host checked the type)
      ux = gux * (1 - nx);
      uy = guy * (1 - ny);
      vx = gvx * (1 - nx);
      vy = gvy * (1 - ny);
    }
    const double p = rho / 3.0 * gamma;
    dr = dr + ((p - visc_g * ux) * nx - visc_g * uy * ny) * area;
    li = li + (visc_g * vx * nx - (p - visc_g * vy) * ny) * area;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    dr += __shfl_down_sync(0xffffffffu, dr, s);
    li += __shfl_down_sync(0xffffffffu, li, s);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = dr;
    red[threadIdx.x >> 5][1] = li;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double d = 0.0, l = 0.0;
    for (int w = 0; w < kWallBlock / 32; w++) {
      d += red[w][0];
      l += red[w][1];
    }
    out[0] = d;
    out[1] = l;
  }
}

inline int blocks_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

// The seven branch decisions of each unique face record of the compact
// layout and the area factors face_flux forms per face without it.
template <int FL>
__global__ void k_record_sides(const void* frec0, const void* frec1, const void* frec2, double cd,
                               int n, int32_t* out, double2* relax) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const d4 f0 = ld4(frec0, r), f1 = ld4(frec1, r), f2 = ld4(frec2, r);
    const double cA = __dmul_rn(f0.w, cd);
    relax[r] = make_double2(__dmul_rn(__dadd_rn(1.0, -f2.w), cA), __dmul_rn(f2.w, cA));
    const double nv[3] = {f0.x, f0.y, f0.z};
    const unsigned sides = face_sides<FL>(nv, f1.x);
    out[r] = (int32_t)(sides | face_kind<FL>(f0, f1, f2, sides) << kKindShift);
  }
}

}  // namespace

void launch_record_sides(const void* frec0, const void* frec1, const void* frec2, double cd, int n,
                         int flavour, int32_t* out, double* relax, cudaStream_t s) {
  if (n <= 0) return;
  const int nb = (int)blocks_for(n, kBlock);
  double2* rl = reinterpret_cast<double2*>(relax);
  if (flavour == PLFBS_FLAVOUR_CPU_SOLVER)
    k_record_sides<1><<<nb, kBlock, 0, s>>>(frec0, frec1, frec2, cd, n, out, rl);
  else
    k_record_sides<0><<<nb, kBlock, 0, s>>>(frec0, frec1, frec2, cd, n, out, rl);
}

void launch_gradient(const KernelArgs& a, int precision, cudaStream_t s) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_gradient32(a, s);
  const int nb = blocks_for(a.C, kBlock);
  const bool cw = a.compact && a.wtab;
  if (a.flavour == PLFBS_FLAVOUR_CPU_SOLVER) {
    if (cw)
      k_gradient<1, true><<<nb, kBlock, 0, s>>>(a);
    else
      k_gradient<1, false><<<nb, kBlock, 0, s>>>(a);
  } else {
    if (cw)
      k_gradient<0, true><<<nb, kBlock, 0, s>>>(a);
    else
      k_gradient<0, false><<<nb, kBlock, 0, s>>>(a);
  }
}
int prepare_flux_tma() {
  static std::atomic<int> tma_resident[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  int r = tma_resident[dev].load(std::memory_order_relaxed);
  if (r <= 0) {
    int per_sm = 0, sms = 0;
    cudaFuncSetAttribute(k_flux_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, kTmaSmem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flux_tma, kTmaThreads, kTmaSmem) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        per_sm <= 0 || sms <= 0) {
      per_sm = 1;
      sms = 148;
    }
    r = per_sm * sms;
    tma_resident[dev].store(r, std::memory_order_relaxed);
  }
  return r;
}

void launch_flux(const KernelArgs& a, int precision, cudaStream_t s) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_flux32(a, s);
  static std::atomic<int> resident[kMaxDevices];
  const bool cr = a.compact && a.face_rec;
  if (a.flavour == PLFBS_FLAVOUR_CPU_SOLVER) {
    static std::atomic<int> cpu_resident[kMaxDevices], cpu_cr_resident[kMaxDevices];
    if (cr)
      k_flux<1, true><<<persistent_blocks(k_flux<1, true>, kFluxBlock, a.F, cpu_cr_resident),
                        kFluxBlock, 0, s>>>(a, 0, a.F);
    else
      k_flux<1, false><<<persistent_blocks(k_flux<1, false>, kFluxBlock, a.F, cpu_resident),
                         kFluxBlock, 0, s>>>(a, 0, a.F);
    return;
  }
  if (!a.flux_maps || a.Fi == 0) {
    static std::atomic<int> cr_resident[kMaxDevices];
    if (cr)
      k_flux<0, true><<<persistent_blocks(k_flux<0, true>, kFluxBlock, a.F, cr_resident),
                        kFluxBlock, 0, s>>>(a, 0, a.F);
    else
      k_flux<0, false><<<persistent_blocks(k_flux<0, false>, kFluxBlock, a.F, resident),
                         kFluxBlock, 0, s>>>(a, 0, a.F);
    return;
  }
  // internal faces through the TMA-staged kernel, boundary faces (the last
  // F - Fi of the face order) through the per-thread one
  const int r = prepare_flux_tma();
  const int tiles = (a.Fi + kTmaFaces - 1) / kTmaFaces;
  k_flux_tma<<<tiles < r ? tiles : r, kTmaThreads, kTmaSmem, s>>>(a, *a.flux_maps);
  if (a.F > a.Fi) {
    static std::atomic<int> bnd_resident[kMaxDevices];
    k_flux<0, false><<<persistent_blocks(k_flux<0, false>, kFluxBlock, a.F - a.Fi, bnd_resident),
                       kFluxBlock, 0, s>>>(a, a.Fi, a.F);
  }
}
template <int RK>
static void launch_update_rk(const KernelArgs& a, cudaStream_t s) {
  const int nb = blocks_for(a.C, kBlock);
  if (a.K2 <= 4)
    k_update<RK, 4><<<nb, kBlock, 0, s>>>(a);
  else if (a.K2 <= 6)
    k_update<RK, 6><<<nb, kBlock, 0, s>>>(a);
  else if (a.K2 <= 8)
    k_update<RK, 8><<<nb, kBlock, 0, s>>>(a);
  else
    k_update<RK, 0><<<nb, kBlock, 0, s>>>(a);
}
void launch_update(const KernelArgs& a, int precision, int rk, cudaStream_t s, bool finish) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_update32(a, rk, s, finish);
  switch (rk) {
    case 0: launch_update_rk<0>(a, s); break;
    case 1: launch_update_rk<1>(a, s); break;
    case 2: launch_update_rk<2>(a, s); break;
    default:
      launch_update_rk<3>(a, s);
      if (finish) k_finish<<<1, kFinishBlock, 0, s>>>(a);
      break;
  }
}
void launch_finish(const KernelArgs& a, int precision, cudaStream_t s) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_finish32(a, s);
  k_finish<<<1, kFinishBlock, 0, s>>>(a);
}
void launch_seed(const KernelArgs& a, int precision, bool conserved, cudaStream_t s) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_seed32(a, conserved, s);
  if (conserved)
    k_seed<true><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
  else
    k_seed<false><<<blocks_for(a.C, kBlock), kBlock, 0, s>>>(a);
}
void launch_ibm(const KernelArgs& a, int precision, cudaStream_t s) {
  if (precision == PLFBS_FP32_DEVIATION) return launch_ibm32(a, s);
  if (a.N > 0) k_ibm<<<blocks_for(8LL * a.N, kIbmBlock), kIbmBlock, 0, s>>>(a);
}

void launch_wall_forces(const KernelArgs& a, int precision, const int* walls, int n,
                        double visc_gamma, double gamma, double* out, cudaStream_t s) {
  k_wall_forces<<<1, kWallBlock, 0, s>>>(a, walls, n, precision == PLFBS_FP32_DEVIATION ? 1 : 0,
                                          visc_gamma, gamma, out);
}

}  // namespace plfbs
