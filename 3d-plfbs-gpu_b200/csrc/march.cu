// The whole time march of a small mesh as one cooperative kernel (FP64 and the
// FP32 deviation form): every SM keeps one tile of cells (tiles.cu) and the grid
// walks the steps, with a grid-wide barrier after each RK stage. Per stage a
// block computes
//   the gradients of its own cells and of the halo cells across its cut faces
//   (k_gradient), into shared memory,
//   the fluxes of all faces of its own cells (k_flux), into shared memory,
//   gather, body force and RK stage of its own cells (k_update);
// stages alternate between two state arrays, since other blocks still read the
// input, and a step's four stages end where they began. The residual sums, the
// convergence test (k_finish) and the body's nodes (k_ibm) are part of the
// walk.
//
// Why: on meshes of up to some ten thousand cells the 14 kernels of a step cost
// their launch, cold instruction and constant caches and three dependent rounds
// of loads each, 4 to 6 us at any size, while their work is a fraction of a
// microsecond. Here a stage costs one barrier and one round of gathers, the
// indices of the next stage are loaded before the barrier, and gradients and
// fluxes never leave the SM; the price, cut faces and halo gradients computed
// by both neighbours, is paid by SMs that were idle.
//
// The arithmetic and the order of every sum are those of the three kernels, so
// a march and the same stages run one by one give the same bits (but for the
// atomic sums of a body's forces in cells that several of its nodes reach).
//
// Every wait is bounded: a block that gives up sets the fault and halt flags
// and leaves, as do then the others. Between steps the march gives way to other
// calls that want its SMs (device_share.hpp).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device_share.hpp"
#include "flux_core.cuh"
#include "flux_core32.cuh"
#include "ibm_core.cuh"
#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

constexpr int kSpinLimit = 1 << 22;

// Compact tables of up to this many records and weight sets are copied to
// shared memory (ST): a barrier's acquire empties L1, so that every stage would
// fetch them from L2 again.
constexpr int kTableMax = 32;
constexpr int kRecRow = 16;  // a record's row there

// The FP64 and FP32 forms of what the kernel calls.
template <int FL_, bool CR_, bool CW_, bool ST_ = false>
struct Form64 {
  static constexpr int FL = FL_;
  static constexpr bool CR = CR_, CW = CW_, ST = ST_;
  using T = double;
  using V = d4;
  static __device__ __forceinline__ V ldrw(const void* p, long long i) { return ld4rw(p, i); }
  static __device__ __forceinline__ void st(void* p, long long i, const V& v) { st4(p, i, v); }
  static __device__ __forceinline__ T fma_(T a, T b, T c) { return fma(a, b, c); }
  static __device__ __forceinline__ int types(const KernelArgs& a, int b) {
    return (int)__ldg(reinterpret_cast<const double*>(a.bc3) + 4LL * b + 3);
  }
  static __device__ __forceinline__ V ghost(const V& q, const V& tgt, int types) {
    return ghost_state<FL>(q, tgt, types);
  }
  // ST: record r's row of the shared tables: n, A | dt, t1 | t2, tau | omA, tA
  static __device__ __forceinline__ void record(const KernelArgs& a, int r, V rec[3]) {
    rec[0] = ld4(CR ? a.frec0 : a.face0, r);
    rec[1] = ld4(CR ? a.frec1 : a.face1, r);
    rec[2] = ld4(CR ? a.frec2 : a.face2, r);
  }
  static __device__ __forceinline__ V row(const T* tab, int r, int k) {
    const double2* p = reinterpret_cast<const double2*>(tab + r * kRecRow + 4 * k);
    const double2 x = p[0], y = p[1];
    return V{x.x, x.y, y.x, y.y};
  }
  static __device__ __forceinline__ void put_record(const KernelArgs& a, int r, T* p) {
    const V f0 = ld4(a.frec0, r), f1 = ld4(a.frec1, r), f2 = ld4(a.frec2, r);
    const V v[3] = {f0, f1, f2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      p[4 * k] = v[k].x;
      p[4 * k + 1] = v[k].y;
      p[4 * k + 2] = v[k].z;
      p[4 * k + 3] = v[k].w;
    }
    const double* w = a.frec_relax + 2 * (size_t)r;
    p[12] = w[0];
    p[13] = w[1];
  }
  static __device__ __forceinline__ V flux(const KernelArgs& a, const T* tab, const V rec[3],
                                           int f, int r, unsigned sides, const V& qo, const V& qn,
                                           T g1[12], T g2[12], bool ghost_side) {
    const V f1 = ST ? row(tab, r, 1) : rec[1], f2 = ST ? row(tab, r, 2) : rec[2];
    const T t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
    T si[4], sn[4], sc[4];
    if (ghost_side)
      boundary_sides<FL>(a, f - a.Fi, t1, t2, qo, g1, g2, si, sn, sc);
    else
      interior_sides(t1, t2, qo, qn, g1, g2, si, sn, sc);
    double R, m[3], P[6];
    face_moments<FL>(a.eq_k0, a.eq_k1, f1.x, sides, si, sn, sc, g1, g2, R, m, P);
    const V f0 = ST ? row(tab, r, 0) : rec[0];
    const double n[3] = {f0.x, f0.y, f0.z};
    double omA, tA;  // as face_flux forms them
    if (ST) {
      const double2 w = *reinterpret_cast<const double2*>(tab + r * kRecRow + 12);
      omA = w.x;
      tA = w.y;
    } else {
      const double cA = __dmul_rn(f0.w, a.eq_cd);
      omA = __dmul_rn(__dadd_rn(1.0, -f2.w), cA);
      tA = __dmul_rn(f2.w, cA);
    }
    return flux_of_moments(a, R, m, P, n, f0.w, omA, tA);
  }
  template <int RK>
  static __device__ __forceinline__ void rk(const KernelArgs& a, const V& t0, const V& t1,
                                            const T R[4], V& q, V& acc) {
    rk_stage<RK>(a.dt, t0, t1, R, q, acc);
  }
  static __device__ __forceinline__ bool bad(const KernelArgs&, const V& acc) {
    return !(acc.w <= 1000.0);  // the CPU solver's divergence test, Solver.cpp:448-493
  }
  static __device__ __forceinline__ T* force(const KernelArgs& a, int c) {
    return c == 0 ? a.force_x : c == 1 ? a.force_y : a.force_z;
  }
  static __device__ __forceinline__ T pressure(const KernelArgs& a) { return a.pressure_gradient; }
  static __device__ __forceinline__ void ibm(const KernelArgs& a, int k) { ibm_thread(a, k); }
};

template <bool CR_, bool CW_, bool ST_ = false>
struct Form32 {
  static constexpr bool CR = CR_, CW = CW_, ST = ST_;
  using T = float;
  using V = f4;
  static __device__ __forceinline__ V ldrw(const void* p, long long i) { return ldf_rw(p, i); }
  static __device__ __forceinline__ void st(void* p, long long i, const V& v) { stf(p, i, v); }
  static __device__ __forceinline__ T fma_(T a, T b, T c) { return fmaf(a, b, c); }
  static __device__ __forceinline__ int types(const KernelArgs& a, int b) {
    return (int)__ldg(reinterpret_cast<const float*>(a.bc3) + 4LL * b + 3);
  }
  static __device__ __forceinline__ V ghost(const V& q, const V& tgt, int types) {
    return ghost_state32(q, tgt, types);
  }
  static __device__ __forceinline__ void record(const KernelArgs& a, int r, V rec[3]) {
    rec[0] = ldf(CR ? a.frec0 : a.face0, r);
    rec[1] = ldf(CR ? a.frec1 : a.face1, r);
    rec[2] = ldf(CR ? a.frec2 : a.face2, r);
  }
  static __device__ __forceinline__ V row(const T* tab, int r, int k) {
    const float4 x = *reinterpret_cast<const float4*>(tab + r * kRecRow + 4 * k);
    return V{x.x, x.y, x.z, x.w};
  }
  static __device__ __forceinline__ void put_record(const KernelArgs& a, int r, T* p) {
    const V v[3] = {ldf(a.frec0, r), ldf(a.frec1, r), ldf(a.frec2, r)};
#pragma unroll
    for (int k = 0; k < 3; k++)
      *reinterpret_cast<float4*>(p + 4 * k) = make_float4(v[k].x, v[k].y, v[k].z, v[k].w);
  }
  static __device__ __forceinline__ V flux(const KernelArgs& a, const T* tab, const V rec[3],
                                           int f, int r, unsigned sides, const V& qo, const V& qn,
                                           T g1[12], T g2[12], bool ghost_side) {
    const V f0 = ST ? row(tab, r, 0) : rec[0], f1 = ST ? row(tab, r, 1) : rec[1],
            f2 = ST ? row(tab, r, 2) : rec[2];
    const T n[3] = {f0.x, f0.y, f0.z}, t1[3] = {f1.y, f1.z, f1.w}, t2[3] = {f2.x, f2.y, f2.z};
    T si[4], sn[4], sc[4];
    if (ghost_side)
      boundary_sides32(a, f - a.Fi, t1, t2, qo, g1, g2, si, sn, sc);
    else
      interior_sides32(t1, t2, qo, qn, g1, g2, si, sn, sc);
    return face_flux32(a, n, f0.w, f2.w, sides, f1.x, si, sn, sc, g1, g2);
  }
  template <int RK>
  static __device__ __forceinline__ void rk(const KernelArgs& a, const V& t0, const V& t1,
                                            const T R[4], V& q, V& acc) {
    rk_stage32<RK>((float)a.dt, a.rho0f, t0, t1, R, q, acc);
  }
  static __device__ __forceinline__ bool bad(const KernelArgs& a, const V& acc) {
    return !(__fadd_rn(a.rho0f, acc.w) <= 1000.0f);
  }
  static __device__ __forceinline__ T* force(const KernelArgs& a, int c) {
    return c == 0 ? a.fforce_x : c == 1 ? a.fforce_y : a.fforce_z;
  }
  static __device__ __forceinline__ T pressure(const KernelArgs& a) {
    return __fmul_rn((float)a.pressure_gradient, a.inv_uref_f);
  }
  static __device__ __forceinline__ void ibm(const KernelArgs& a, int k) { ibm_thread32(a, k); }
};

// Shared-memory row of a cell: state (u, v, w, rho) and gradient (12), padded so
// that a warp's 16-byte accesses to consecutive rows meet no bank twice (FP64
// 144 B, FP32 80 B).
template <typename T>
constexpr int row_size() {
  return sizeof(T) == 8 ? 18 : 20;
}
__device__ __forceinline__ d4 row4(const double* p) {
  const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
  return d4{x.x, x.y, y.x, y.y};
}
__device__ __forceinline__ f4 row4(const float* p) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  return f4{x.x, x.y, x.z, x.w};
}
__device__ __forceinline__ void row4(double* p, const d4& v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v.x, v.y);
  reinterpret_cast<double2*>(p)[1] = make_double2(v.z, v.w);
}
__device__ __forceinline__ void row4(float* p, const f4& v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.x, v.y, v.z, v.w);
}

// What a thread keeps of its own cell over the march, in shared memory: the RK
// accumulators t0 and t1 and 1 / volume (an odd row, word accesses).
constexpr int kOwn = 9;

template <typename Fm, int RK>
__device__ __forceinline__ void stage_update(const KernelArgs& a, int i, const typename Fm::T R[4],
                                             typename Fm::T* own, void* out, double sq[4],
                                             bool& bad) {
  using V = typename Fm::V;
  const V t0{own[0], own[1], own[2], own[3]}, t1{own[4], own[5], own[6], own[7]};
  V q, acc;
  Fm::template rk<RK>(a, t0, t1, R, q, acc);
  if (RK == 3) {
    sq[0] = (double)R[3] * R[3];
    sq[1] = (double)R[0] * R[0];
    sq[2] = (double)R[1] * R[1];
    sq[3] = (double)R[2] * R[2];
    bad = Fm::bad(a, acc);
  }
  typename Fm::T* p = own + (RK == 3 ? 0 : 4);  // the next step starts from the accumulator
  p[0] = acc.x;
  p[1] = acc.y;
  p[2] = acc.z;
  p[3] = acc.w;
  Fm::st(out, i, q);
}

// The tile's tables, each in shared memory where it fits (a barrier's acquire
// empties L1, and a load from L2 takes some 1,200 cycles here).
template <typename Fm>
struct Tables {
  const int32_t *cell, *nbr, *wset;
  const uint32_t* ij;
  const int32_t* id;  // record (compact layout) or device face with branch bits
  const uint16_t* slot;
};

// A local cell's device index, stencil neighbours and weight set.
constexpr int kNbrPre = 6;
struct LocalCell {
  int cell, wset, nb[kNbrPre];
};
template <typename Fm>
__device__ __forceinline__ LocalCell local_cell(const Tables<Fm>& b, int K, int SC, int l) {
  LocalCell x;
  const bool in = l < SC;
  x.cell = in ? b.cell[l] : -1;
#pragma unroll
  for (int k = 0; k < kNbrPre; k++) x.nb[k] = in && k < K ? b.nbr[k * SC + l] : -1;
  x.wset = Fm::CW && in ? b.wset[l] : 0;
  return x;
}

// Gradient of local cell l into its shared-memory row. One round of loads: the
// own state, of each of up to KU stencil slots the neighbour's state (a ghost's
// boundary target and types, the own state again for an empty slot) and, unless
// they are in shared memory (wt), the weights.
template <typename Fm, int KU>
__device__ __forceinline__ void stage_gradient(const KernelArgs& a, const Tables<Fm>& b,
                                               const LocalCell& x, int l, const void* in,
                                               const typename Fm::T* wt, typename Fm::T* S) {
  using T = typename Fm::T;
  using V = typename Fm::V;
  const int i = x.cell;
  if (i < 0) return;  // the list's padding
  const V* st = static_cast<const V*>(in);
  const V qi = Fm::ldrw(st, i);
  V qj[KU];
  int types[KU];
#pragma unroll
  for (int k = 0; k < KU; k++) {
    const int j = x.nb[k];
    const bool ghost = j >= a.C;
    qj[k] = Fm::ldrw(ghost ? static_cast<const V*>(a.bc1) : st, ghost ? j - a.C : j < 0 ? i : j);
    types[k] = ghost ? Fm::types(a, j - a.C) : 0;
  }
  const T* wrow = Fm::CW ? (Fm::ST ? wt : static_cast<const T*>(a.wtab)) + x.wset * a.K * 3 : nullptr;
  auto weights = [&](int k, T w[3]) {
    const long long s = (long long)k * a.C + i;
    w[0] = Fm::ST ? wrow[3 * k] : Fm::CW ? __ldg(wrow + 3 * k) : __ldg(static_cast<const T*>(a.st_wx) + s);
    w[1] = Fm::ST ? wrow[3 * k + 1] : Fm::CW ? __ldg(wrow + 3 * k + 1) : __ldg(static_cast<const T*>(a.st_wy) + s);
    w[2] = Fm::ST ? wrow[3 * k + 2] : Fm::CW ? __ldg(wrow + 3 * k + 2) : __ldg(static_cast<const T*>(a.st_wz) + s);
  };
  T w[Fm::ST ? 1 : KU][3];
  if (!Fm::ST) {
#pragma unroll
    for (int k = 0; k < KU; k++)
      if (k < a.K) weights(k, w[Fm::ST ? 0 : k]);
  }
  T g[12];
#pragma unroll
  for (int k = 0; k < 12; k++) g[k] = T(0);
  auto add = [&](const V& q, const T u[3]) {
    const T d[4] = {q.w - qi.w, q.x - qi.x, q.y - qi.y, q.z - qi.z};
#pragma unroll
    for (int f = 0; f < 4; f++)
#pragma unroll
      for (int c = 0; c < 3; c++) g[3 * f + c] = Fm::fma_(u[c], d[f], g[3 * f + c]);
  };
#pragma unroll
  for (int k = 0; k < KU; k++) {
    if (x.nb[k] < 0) continue;
    if (x.nb[k] >= a.C) qj[k] = Fm::ghost(qi, qj[k], types[k]);
    if (Fm::ST) weights(k, w[0]);
    add(qj[k], w[Fm::ST ? 0 : k]);
  }
  for (int k = KU; k < a.K; k++) {  // wider stencils
    const int j = b.nbr[k * a.tiles.SC + l];
    if (j < 0) break;
    T u[3];
    weights(k, u);
    add(j < a.C ? Fm::ldrw(st, j)
                : Fm::ghost(qi, Fm::ldrw(a.bc1, j - a.C), Fm::types(a, j - a.C)), u);
  }
  T* row = S + l * row_size<T>();
  row4(row, qi);
  row4(row + 4, V{g[0], g[1], g[2], g[3]});
  row4(row + 8, V{g[4], g[5], g[6], g[7]});
  row4(row + 12, V{g[8], g[9], g[10], g[11]});
}

// A face's entry, its local cells and branch bits and its record (compact
// layout) or device face; and, without the records in shared memory, the
// record itself, loaded a face ahead.
template <typename Fm>
struct FaceEntry {
  uint32_t ij;
  int32_t id;
  typename Fm::V rec[Fm::ST ? 1 : 3];
};
template <typename Fm>
__device__ __forceinline__ FaceEntry<Fm> face_entry(const KernelArgs& a, const Tables<Fm>& b, int p) {
  FaceEntry<Fm> x;
  x.ij = b.ij[p];
  x.id = b.id[p];
  if (!Fm::ST) Fm::record(a, Fm::CR ? x.id : x.id & 0xfffffff, x.rec);
  return x;
}

template <typename Fm>
__device__ __forceinline__ void stage_flux(const KernelArgs& a, const TileArgs& t, size_t e,
                                           const FaceEntry<Fm>& x, const typename Fm::T* tab,
                                           const typename Fm::T* S, typename Fm::T* X) {
  using T = typename Fm::T;
  using V = typename Fm::V;
  const int lo = x.ij & 2047, ln = x.ij >> 11 & 2047;
  const bool ghost_side = ln == kTileGhost;
  // the branch bits: per record with the FP64 compact layout, else from the
  // entry (its high two with the device face)
  int f = 0;
  unsigned sides;
  if (Fm::ST) {
    sides = __float_as_uint(reinterpret_cast<const float*>(tab + x.id * kRecRow + 14)[0]);
    if (ghost_side) f = __ldg(t.fid + e) & 0xfffffff;
  } else if (Fm::CR && sizeof(T) == 8) {
    sides = (unsigned)__ldg(a.frec_sides + x.id);
    if (ghost_side) f = __ldg(t.fid + e) & 0xfffffff;
  } else {
    const uint32_t v = Fm::CR ? (uint32_t)__ldg(t.fid + e) : (uint32_t)x.id;
    f = (int)(v & 0xfffffffu);
    sides = x.ij >> 22 | v >> 28 << 10;
  }
  const int r = Fm::CR ? x.id : f;
  const T* ro = S + lo * row_size<T>();
  const T* rn = S + (ghost_side ? lo : ln) * row_size<T>();
  const V qo = row4(ro), qn = row4(rn);
  T g1[12], g2[12];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const V x = row4(ro + 4 + 4 * k), y = row4(rn + 4 + 4 * k);
    g1[4 * k] = x.x; g1[4 * k + 1] = x.y; g1[4 * k + 2] = x.z; g1[4 * k + 3] = x.w;
    g2[4 * k] = y.x; g2[4 * k + 1] = y.y; g2[4 * k + 2] = y.z; g2[4 * k + 3] = y.w;
  }
  const V y = Fm::flux(a, tab, x.rec, f, r, sides, qo, qn, g1, g2, ghost_side);
  X[0] = y.x;
  X[t.SF] = y.y;
  X[2 * t.SF] = y.z;
  X[3 * t.SF] = y.w;
}

// Grid-wide barrier in two halves. The counter only grows; `target` is the
// arrivals after which a wait passes.
__device__ __forceinline__ void grid_arrive(unsigned* bar) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ __forceinline__ bool grid_wait(const unsigned* bar, unsigned target) {
  bool ok = true;
  if (threadIdx.x == 0) {
    ok = false;
    for (int i = 0; i < kSpinLimit && !ok; i++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      ok = (int)(v - target) >= 0;
    }
  }
  return __syncthreads_and(ok);
}

// The step's norms from the tiles' sums, as k_finish (same order of additions);
// every block forms them and takes the same decision, block 0 records the
// step. Returns whether the march ends: the context halts, or it gives way.
__device__ __forceinline__ bool step_norms(const KernelArgs& a, long long step) {
  __shared__ double red[kMaxTiles / 32][4];
  __shared__ int stop;
  __shared__ bool bad, give_way;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // by a warp that loads no sums: beside them, not before (0.2 to 0.3 us per step)
  if (tid == (int)blockDim.x - 1) {
    bad = *(volatile const int*)&a.stats->diverged != 0;
    give_way = *(volatile const unsigned*)(a.grid_bar + 1) != 0;
  }
  if (tid < kMaxTiles) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      double v = tid < a.tiles.n ? a.partial[4 * tid + c] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][c] = v;
    }
  }
  __syncthreads();
  if (warp == 0) {
    double rms = 0.0;
    if (lane < 4) {
      double tot = 0.0;
      for (int w = 0; w < kMaxTiles / 32; w++) tot += red[w][lane];
      rms = sqrt(tot / (double)a.C) * (lane == 0 ? a.inv_ref_rho : a.inv_ref_mom);
    }
    const double rho = __shfl_sync(0xffffffffu, rms, 0), u = __shfl_sync(0xffffffffu, rms, 1),
                 v = __shfl_sync(0xffffffffu, rms, 2), w = __shfl_sync(0xffffffffu, rms, 3);
    const double me = fmax(fmax(w, u), v);  // residuals::max_error
    const bool diverged = bad || !(me == me) || !(rho == rho), converged = me < a.tolerance;
    if (lane == 0) {
      stop = diverged || converged || give_way;
      if (blockIdx.x == 0) {
        DevStats* st = a.stats;
        double* h = st->history[step % kHistoryCap];
        h[0] = st->last[0] = (double)step;
        h[1] = st->last[1] = me;
        h[2] = st->last[2] = rho;
        h[3] = st->last[3] = u;
        h[4] = st->last[4] = v;
        h[5] = st->last[5] = w;
        st->steps = step + 1;
        if (diverged) st->diverged = 1;
        if (converged) {
          st->converged = 1;
          st->converged_step = step;
        }
        if (diverged || converged) st->halt = 1;
      }
    }
  }
  __syncthreads();
  return stop != 0;
}

// Marches to time step `end` of the run. `wanted` (null: no look) is the sum of
// SMs wanted on the device (device_share.hpp); the march gives way, at the end of a
// step, once it no longer fits beside the others.
template <typename Fm, int NT>
__global__ void __launch_bounds__(NT, 1)
    k_march(const KernelArgs a, const long long end, const int* wanted, const int sms) {
  using T = typename Fm::T;
  using V = typename Fm::V;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kTileMaxOwn / 32][4];
  const TileArgs& t = a.tiles;
  constexpr int kRow = row_size<T>();
  T* S = reinterpret_cast<T*>(smem);
  T* X = S + (size_t)t.SC * kRow;   // flux components, [4][SF]
  T* tab = X + 4 * (size_t)t.SF;    // ST: record rows, then weight sets
  T* wt = tab + (Fm::ST ? a.n_frec * kRecRow : 0);
  T* own0 = wt + (Fm::ST ? a.n_wset * a.K * 3 : 0);
  const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  if (*(volatile const int*)&a.stats->halt) return;  // the same for every block
  const long long step0 = *(volatile const long long*)&a.stats->steps;
  const int nf = __ldg(t.count + tile).y, own_n = min(t.T, a.C - tile * t.T);
  Tables<Fm> b;
  {
    unsigned char* q = reinterpret_cast<unsigned char*>(own0 + (size_t)t.T * kOwn);
    auto place = [&](const auto* src, int n, int bit) {
      using E = std::remove_const_t<std::remove_pointer_t<decltype(src)>>;
      if (!(t.place & bit)) return src;
      E* dst = reinterpret_cast<E*>(q);
      for (int k = tid; k < n; k += NT) dst[k] = __ldg(src + k);
      q += ((size_t)n * sizeof(E) + 15) / 16 * 16;
      return static_cast<const E*>(dst);
    };
    b.slot = place(static_cast<const uint16_t*>(t.slot + (size_t)tile * a.K2 * t.T), a.K2 * t.T, 1);
    b.ij = place(static_cast<const uint32_t*>(t.ij + (size_t)tile * t.SF), t.SF, 2);
    b.id = place(static_cast<const int32_t*>((Fm::CR ? t.rec : t.fid) + (size_t)tile * t.SF), t.SF, 2);
    b.cell = place(static_cast<const int32_t*>(t.cell + (size_t)tile * t.SC), t.SC, 4);
    b.nbr = place(static_cast<const int32_t*>(t.nbr + (size_t)tile * a.K * t.SC), a.K * t.SC, 4);
    b.wset = Fm::CW ? place(static_cast<const int32_t*>(t.wset + (size_t)tile * t.SC), t.SC, 4)
                    : nullptr;
  }
  for (int u = tid; u < own_n; u += NT) {
    const int i = __ldg(t.cell + (size_t)tile * t.SC + u);
    T* own = own0 + u * kOwn;
    const V t0 = Fm::ldrw(a.t0, i);
    own[0] = t0.x;
    own[1] = t0.y;
    own[2] = t0.z;
    own[3] = t0.w;
    own[8] = __ldg(static_cast<const T*>(a.inv_volume) + i);
  }
  if (Fm::ST) {
    for (int r = tid; r < a.n_frec; r += NT) {
      Fm::put_record(a, r, tab + r * kRecRow);
      reinterpret_cast<float*>(tab + r * kRecRow + 14)[0] =
          __uint_as_float((unsigned)__ldg(a.frec_sides + r));
    }
    for (int k = tid; k < a.n_wset * a.K * 3; k += NT)
      wt[k] = __ldg(static_cast<const T*>(a.wtab) + k);
  }
  __syncthreads();
  unsigned arrived = 0;  // arrivals of all blocks at the barriers so far
  int others = t.n;      // the last look at `wanted`, by one thread
  bool ok = true, stop = false;
  const int nsteps = (int)(end - step0);  // a batch at most
  for (int n = 0; n < nsteps && ok && !stop; n++) {
    if (a.N > 0) {  // the body, before the stages
      for (int k = blockIdx.x * NT + tid; (k & ~31) < 8 * a.N; k += gridDim.x * NT)
        Fm::ibm(a, k);
      grid_arrive(a.grid_bar);  // awaited before the first update
      arrived += gridDim.x;
    }
#pragma unroll 1
    for (int rk = 0; rk < 4; rk++) {
      const void* in = (rk & 1) ? a.state2 : a.state;
      void* out = (rk & 1) ? a.state : a.state2;
      LocalCell lc = local_cell<Fm>(b, a.K, t.SC, tid);
      // the look crosses the host link: on its way through two stages, and every
      // fourth step (each step: 48.5 us instead of 48.0 on 65,536 cells FP32)
      if (rk == 1 && (n & 3) == 0 && wanted && tile == t.n - 1 && tid == NT - 1)
        others = *(volatile const int*)wanted;
      if (rk > 0) {  // the previous stage's states, on every SM
        ok = grid_wait(a.grid_bar, arrived);
        if (!ok) break;
      }
      for (int l = tid; l < t.SC; l += NT) {
        const LocalCell next = local_cell<Fm>(b, a.K, t.SC, l + NT);
        if (a.K <= 4)
          stage_gradient<Fm, 4>(a, b, lc, l, in, wt, S);
        else
          stage_gradient<Fm, kNbrPre>(a, b, lc, l, in, wt, S);
        lc = next;
      }
      FaceEntry<Fm> fe = face_entry<Fm>(a, b, min(tid, t.SF - 1));
      __syncthreads();
#pragma unroll 1
      for (int p = tid; p < nf; p += NT) {
        const FaceEntry<Fm> next = face_entry<Fm>(a, b, min(p + NT, t.SF - 1));
        stage_flux<Fm>(a, t, (size_t)tile * t.SF + p, fe, tab, S, X + p);
        fe = next;
      }
      if (rk == 0 && a.N > 0) {
        ok = grid_wait(a.grid_bar, arrived);  // the body's forces; also a block barrier
        if (!ok) break;
      } else {
        __syncthreads();
      }
      // update of the own cells, a warp's 32 at a time; in the last stage their
      // squared residuals' sums, as k_update's
      bool bad = false;
#pragma unroll 1
      for (int u = tid; (u & ~31) < own_n; u += NT) {
        double sq[4] = {0.0, 0.0, 0.0, 0.0};
        if (u < own_n) {
          const int i = b.cell[u];
          T *fx = Fm::force(a, 0), *fy = Fm::force(a, 1), *fz = Fm::force(a, 2);
          T fc[3] = {Fm::pressure(a), T(0), T(0)};
          if (fx) {
            fc[0] = fx[i];
            fc[1] = fy[i];
            fc[2] = fz[i];
          }
          T r[4] = {T(0), T(0), T(0), T(0)};
          for (int k = 0; k < a.K2; k++) {
            const unsigned s = b.slot[k * t.T + u];
            if (s == 0xffffu) break;
            const T* x = X + (s >> 1);
            const T sg = (s & 1) ? T(1) : T(-1);
#pragma unroll
            for (int c = 0; c < 4; c++) r[c] = Fm::fma_(sg, x[c * t.SF], r[c]);
          }
          T* own = own0 + u * kOwn;
          const T iv = own[8];
          const T R[4] = {Fm::fma_(r[0], iv, fc[0]), Fm::fma_(r[1], iv, fc[1]),
                          Fm::fma_(r[2], iv, fc[2]), r[3] * iv};
          switch (rk) {
            case 0: stage_update<Fm, 0>(a, i, R, own, out, sq, bad); break;
            case 1: stage_update<Fm, 1>(a, i, R, own, out, sq, bad); break;
            case 2: stage_update<Fm, 2>(a, i, R, own, out, sq, bad); break;
            default:
              stage_update<Fm, 3>(a, i, R, own, out, sq, bad);
              if (fx) {  // the last reader of this step's force resets it for the body
                fx[i] = Fm::pressure(a);
                fy[i] = T(0);
                fz[i] = T(0);
              }
          }
        }
        if (rk == 3) {
#pragma unroll
          for (int c = 0; c < 4; c++) {
            double v = sq[c];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[u >> 5][c] = v;
          }
        }
      }
      if (rk == 3) {  // and the tile's, as k_finish's
        const int any_bad = __syncthreads_or(bad);
        if (tid < 4) {
          double v = 0.0;
          for (int w = 0; 32 * w < own_n; w++) v += red[w][tid];
          a.partial[4 * tile + tid] = v;
        }
        if (tid == 0 && any_bad) a.stats->diverged = 1;
        if (tile == t.n - 1 && tid == NT - 1 && !march_fits(others, t.n, sms))
          *(volatile unsigned*)(a.grid_bar + 1) = 1;
      }
      grid_arrive(a.grid_bar);
      arrived += gridDim.x;
    }
    if (!ok) break;
    ok = grid_wait(a.grid_bar, arrived);
    if (ok) stop = step_norms(a, step0 + n);
  }
  // what the context keeps between marches: the accumulators, and the ghosts of
  // the last stage's input state as k_gradient leaves them
  for (int u = tid; u < own_n; u += NT) {
    const T* own = own0 + u * kOwn;
    Fm::st(a.t0, b.cell[u], V{own[0], own[1], own[2], own[3]});
    const V qi = row4(S + u * kRow);
    for (int k = 0; k < a.K; k++) {
      const int j = b.nbr[k * t.SC + u];
      if (j >= a.C)
        Fm::st(a.state, j, Fm::ghost(qi, Fm::ldrw(a.bc1, j - a.C), Fm::types(a, j - a.C)));
    }
  }
  if (!ok && tid == 0) {
    atomicExch(&a.stats->fault, 1);
    atomicExch(&a.stats->halt, 1);
  }
}

// call(form) for the instance a context takes.
template <typename Call>
auto with_form(const KernelArgs& a, int precision, Call call) {
  const bool cr = a.compact && a.face_rec, cw = a.compact && a.wtab, st = cr && cw && a.tiles.tables;
  if (precision == PLFBS_FP32_DEVIATION) {
    if (st) return call(Form32<true, true, true>{});
    if (cr) return cw ? call(Form32<true, true>{}) : call(Form32<true, false>{});
    return cw ? call(Form32<false, true>{}) : call(Form32<false, false>{});
  }
  if (a.flavour == PLFBS_FLAVOUR_CPU_SOLVER) {
    if (st) return call(Form64<1, true, true, true>{});
    if (cr) return cw ? call(Form64<1, true, true>{}) : call(Form64<1, true, false>{});
    return cw ? call(Form64<1, false, true>{}) : call(Form64<1, false, false>{});
  }
  if (st) return call(Form64<0, true, true, true>{});
  if (cr) return cw ? call(Form64<0, true, true>{}) : call(Form64<0, true, false>{});
  return cw ? call(Form64<0, false, true>{}) : call(Form64<0, false, false>{});
}

// Threads of a block, one block per SM. FP64 with shared records 512 (128
// registers: 65,536 cells 67 us per step, 71 with 384 threads, 75 with 256);
// with records read per face 256, whose 255 registers hold the next face's
// records (73,002 tetrahedra 93 us with 512 threads, which spill, 81 with 256);
// FP32 512 (65,536 cells 48 us, 53 with 768).
template <typename Fm>
constexpr int march_threads() {
  return sizeof(typename Fm::T) == 8 && !Fm::ST ? 256 : 512;
}

}  // namespace

// Dynamic shared memory of a block (0: it does not fit in `most`) and the tables
// that go there beside the rows, in the order of what their loads cost.
int march_smem(const KernelArgs& a, int precision, int most, TileArgs& t) {
  const size_t e = precision == PLFBS_FP32_DEVIATION ? 4 : 8;
  size_t n = e * ((size_t)t.SC * (e == 8 ? row_size<double>() : row_size<float>()) +
                  4 * (size_t)t.SF + (size_t)t.T * kOwn);
  t.tables = a.face_rec && a.wtab && a.n_frec <= kTableMax && a.n_wset <= kTableMax && a.K <= 8;
  if (t.tables) n += e * ((size_t)a.n_frec * kRecRow + (size_t)a.n_wset * a.K * 3);
  n = (n + 15) / 16 * 16;
  auto up = [](size_t b) { return (b + 15) / 16 * 16; };
  const size_t table[3] = {up(2 * (size_t)a.K2 * t.T), 2 * up(4 * (size_t)t.SF),
                           2 * up(4 * (size_t)t.SC) + up(4 * (size_t)a.K * t.SC)};
  t.place = 0;
  for (int k = 0; k < 3; k++)
    if (n + table[k] <= (size_t)most) {
      n += table[k];
      t.place |= 1 << k;
    }
  return n <= (size_t)most ? (int)n : 0;
}

// The attribute belongs to the kernel on the device, not to a context: threads
// launch the same instance with tiles of different sizes, so every context sets
// the same value, the device's limit. `resident`: the blocks that the device holds
// at once; a cooperative launch of more is refused.
cudaError_t prepare_march(const KernelArgs& a, int precision, int most, int sms, int* resident) {
  cudaError_t e = cudaSuccess;
  KernelArgs args = a;
  *resident = 1 << 30;
  for (int k = 0; k < 2 && e == cudaSuccess; k++) {
    e = with_form(args, precision, [&](auto f) {
      using Fm = decltype(f);
      constexpr int NT = march_threads<Fm>();
      int per_sm = 0;
      cudaError_t err = cudaFuncSetAttribute(
          k_march<Fm, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (err == cudaSuccess)
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_march<Fm, NT>, NT,
                                                            (size_t)a.tiles.smem);
      *resident = std::min(*resident, per_sm * sms);
      return err;
    });
    args.compact = 0;  // plfbs_set_layout_compression
  }
  return e;
}

cudaError_t launch_march(const KernelArgs& a, int precision, long long end, const int* wanted,
                         int sms, cudaStream_t s) {
  return with_form(a, precision, [&](auto f) {
    using Fm = decltype(f);
    constexpr int NT = march_threads<Fm>();
    const cudaError_t e = cudaMemsetAsync(a.grid_bar, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    KernelArgs args = a;
    void* p[] = {&args, &end, &wanted, &sms};
    return cudaLaunchCooperativeKernel(k_march<Fm, NT>, dim3(a.tiles.n), dim3(NT), p,
                                       (size_t)a.tiles.smem, s);
  });
}

}  // namespace plfbs
