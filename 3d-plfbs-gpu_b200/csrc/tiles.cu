// Cell tiles of the march kernel (march.cu), built on the device at
// create: the cells in the order of a Hilbert curve through their centroids,
// cut into runs of T cells, and for each run the tables its block walks. No
// counterpart in the reference.
//
// The curve keeps a run's cells together in space whatever the caller's
// numbering (512 cells of a uniform box are an 8 x 8 x 8 block), so few faces
// cross between tiles: those are computed by both tiles, and the gradient of a
// cell across such a face (a halo cell) by every tile it borders.
#include <cstdint>

#include "flux_core.cuh"
#include "flux_core32.cuh"
#include "plfbs_internal.hpp"

namespace plfbs {
namespace {

constexpr int kTileBlock = 256;
constexpr int kBoundsBlocks = 128;
constexpr int kSortItems = 4096;  // items per block of the radix sort: 8 warps x 512

// ---------------------------------------------------------------------------
// Hilbert order of the cells
// ---------------------------------------------------------------------------

// Per-block bounds of the centroids and sums of the volumes, in a fixed
// partition and order, so that every context of a mesh gets the same tiles.
__global__ void __launch_bounds__(kTileBlock) k_bounds(int C, const double* ccen,
                                                       const double* vol, double* part) {
  __shared__ double red[kTileBlock][7];
  double v[7] = {1e300, 1e300, 1e300, -1e300, -1e300, -1e300, 0.0};
  for (int i = blockIdx.x * kTileBlock + threadIdx.x; i < C; i += kBoundsBlocks * kTileBlock) {
    for (int c = 0; c < 3; c++) {
      const double x = ccen[3 * (size_t)i + c];
      v[c] = fmin(v[c], x);
      v[3 + c] = fmax(v[3 + c], x);
    }
    v[6] += vol[i];
  }
  for (int c = 0; c < 7; c++) red[threadIdx.x][c] = v[c];
  for (int s = kTileBlock / 2; s > 0; s >>= 1) {
    __syncthreads();
    if (threadIdx.x < s)
      for (int c = 0; c < 7; c++) {
        const double a = red[threadIdx.x][c], b = red[threadIdx.x + s][c];
        red[threadIdx.x][c] = c < 3 ? fmin(a, b) : c < 6 ? fmax(a, b) : a + b;
      }
  }
  if (threadIdx.x < 7) part[7 * blockIdx.x + threadIdx.x] = red[0][threadIdx.x];
}

// part -> box[0..2] the lowest centroid, box[3] the lattice spacing, as a
// whole number of lattice cells per axis that fits `bits` bits: the mean cell
// spacing (a uniform box lands on its own indices), wider where the domain
// needs it.
__global__ void k_box(const double* part, int C, int bits, double* box) {
  double v[7];
  for (int c = 0; c < 7; c++) v[c] = part[c];
  for (int b = 1; b < kBoundsBlocks; b++)
    for (int c = 0; c < 7; c++) {
      const double x = part[7 * b + c];
      v[c] = c < 3 ? fmin(v[c], x) : c < 6 ? fmax(v[c], x) : v[c] + x;
    }
  const double ext = fmax(fmax(v[3] - v[0], v[4] - v[1]), v[5] - v[2]);
  double h = cbrt(v[6] / C);
  const double least = ext / ((1 << bits) - 1);
  if (!(h >= least)) h = least;
  if (!(h > 0.0)) h = 1.0;
  for (int c = 0; c < 3; c++) box[c] = v[c];
  box[3] = h;
}

// Position of lattice point x along the Hilbert curve of `bits` bits per axis
// (the transpose form of J. Skilling, "Programming the Hilbert curve", AIP
// Conf. Proc. 707, 2004).
__device__ uint32_t hilbert(uint32_t x[3], int bits) {
  const uint32_t top = 1u << (bits - 1);
  for (uint32_t q = top; q > 1; q >>= 1) {
    const uint32_t p = q - 1;
    for (int i = 0; i < 3; i++) {
      if (x[i] & q) {
        x[0] ^= p;
      } else {
        const uint32_t t = (x[0] ^ x[i]) & p;
        x[0] ^= t;
        x[i] ^= t;
      }
    }
  }
  x[1] ^= x[0];
  x[2] ^= x[1];
  uint32_t t = 0;
  for (uint32_t q = top; q > 1; q >>= 1)
    if (x[2] & q) t ^= q - 1;
  for (int i = 0; i < 3; i++) x[i] ^= t;
  uint32_t key = 0;
  for (int b = bits - 1; b >= 0; b--)
    for (int i = 0; i < 3; i++) key = key << 1 | (x[i] >> b & 1u);
  return key;
}

__global__ void k_hilbert(int C, const double* ccen, const int32_t* cell_new, const double* box,
                          int bits, uint32_t* key, int32_t* val) {
  const double h = box[3];
  const double hi = (double)((1 << bits) - 1);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C; i += gridDim.x * blockDim.x) {
    uint32_t x[3];
    for (int c = 0; c < 3; c++) {
      const double q = (ccen[3 * (size_t)i + c] - box[c]) / h + 0.5;
      x[c] = (uint32_t)fmin(fmax(q, 0.0), hi);
    }
    const int n = cell_new[i];
    key[n] = hilbert(x, bits);
    val[n] = n;
  }
}

// One stable counting pass of the least-significant-digit radix sort over 8
// key bits: digit counts per block (digit-major), then, after their exclusive
// scan, each block's items to their places in order.
__global__ void __launch_bounds__(kTileBlock) k_digit_count(const uint32_t* key, int n, int shift,
                                                            int nblk, int32_t* count) {
  __shared__ int c[256];
  c[threadIdx.x] = 0;
  __syncthreads();
  const int base = blockIdx.x * kSortItems;
  for (int j = threadIdx.x; j < kSortItems; j += kTileBlock)
    if (base + j < n) atomicAdd(&c[key[base + j] >> shift & 255u], 1);
  __syncthreads();
  count[threadIdx.x * nblk + blockIdx.x] = c[threadIdx.x];
}

__global__ void __launch_bounds__(kTileBlock) k_digit_place(const uint32_t* key, const int32_t* val,
                                                            int n, int shift, int nblk,
                                                            const int32_t* off, const int32_t* wbase,
                                                            uint32_t* key_out, int32_t* val_out) {
  __shared__ int c[8][256];  // per warp: counts, then the next place of each digit
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int w = 0; w < 8; w++) c[w][threadIdx.x] = 0;
  __syncthreads();
  const int first = blockIdx.x * kSortItems + warp * (kSortItems / 8);
  for (int j = lane; j < kSortItems / 8; j += 32)
    if (first + j < n) atomicAdd(&c[warp][key[first + j] >> shift & 255u], 1);
  __syncthreads();
  {
    const int at = threadIdx.x * nblk + blockIdx.x;
    int next = wbase[at / kFaceWindow] + off[at];
    for (int w = 0; w < 8; w++) {
      const int k = c[w][threadIdx.x];
      c[w][threadIdx.x] = next;
      next += k;
    }
  }
  __syncthreads();
  for (int j = 0; j < kSortItems / 8; j += 32) {
    const int i = first + j + lane;
    const bool valid = i < n;
    const uint32_t k = valid ? key[i] : 0;
    const unsigned d = valid ? (k >> shift & 255u) : 256u;
    const unsigned same = __match_any_sync(0xffffffffu, d);
    int at = 0;
    if (valid) at = c[warp][d] + __popc(same & ((1u << lane) - 1u));
    __syncwarp();
    if (valid && lane == __ffs(same) - 1) c[warp][d] += __popc(same);
    __syncwarp();
    if (valid) {
      key_out[at] = k;
      val_out[at] = val[i];
    }
  }
}

__global__ void k_positions(const int32_t* order, int C, int32_t* pos) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < C; p += gridDim.x * blockDim.x)
    pos[order[p]] = p;
}

// ---------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------

// Branch bits of every face, from its own records, as the flux forms them.
template <int FL>
__global__ void k_face_sides(const void* face0, const void* face1, int F, uint16_t* side) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F; f += gridDim.x * blockDim.x) {
    const d4 f0 = ld4(face0, f), f1 = ld4(face1, f);
    const double n[3] = {f0.x, f0.y, f0.z};
    side[f] = (uint16_t)face_sides<FL>(n, f1.x);
  }
}
__global__ void k_face_sides32(const float4* face0, const float4* face1, int F, uint16_t* side) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F; f += gridDim.x * blockDim.x)
    side[f] = (uint16_t)face_sides32(face0[f].x, face0[f].y, face0[f].z,
                                       __fmul_rn(0.001f, face1[f].x));
}

struct TileSource {
  int C, F, Fi, K, K2, T;
  const int32_t* order;   // [C] cell at each position of the curve
  const int32_t* pos;     // [C] its inverse
  const int2* face_ids;
  const int32_t* gather;
  const int32_t* st_nbr;
  const int32_t* face_rec;   // or null
  const int32_t* cell_wset;  // or null
  const uint16_t* side;
};

// Calls use(f, is_neighbour, other, mine): the faces of the tile's own cell i,
// `other` the cell across or -1 at a boundary; each face of the tile is mine
// for exactly one of its cells.
template <typename Use>
__device__ __forceinline__ void for_faces(const TileSource& s, int tile, int i, Use use) {
  for (int k = 0; k < s.K2; k++) {
    const int e = s.gather[(size_t)k * s.C + i];
    if (e < 0) break;
    const int f = e >> 1, nb = e & 1;
    const int2 id = s.face_ids[f];
    const int other = nb ? id.x : id.y;
    if (other >= s.C)
      use(k, f, nb, -1, true);
    else
      use(k, f, nb, other, nb == 0 || s.pos[other] / s.T != tile);
  }
}

// most[0], most[1]: the most faces of a tile and the most faces it shares
// with other tiles.
__global__ void __launch_bounds__(kTileBlock) k_tile_count(const TileSource s, int32_t* most) {
  __shared__ int c[2];
  if (threadIdx.x < 2) c[threadIdx.x] = 0;
  __syncthreads();
  const int tile = blockIdx.x;
  int faces = 0, cut = 0;
  for (int l = threadIdx.x; l < s.T; l += kTileBlock) {
    const int p = tile * s.T + l;
    if (p >= s.C) break;
    for_faces(s, tile, s.order[p], [&](int, int, int, int other, bool mine) {
      faces += mine;
      cut += other >= 0 && s.pos[other] / s.T != tile;
    });
  }
  atomicAdd(&c[0], faces);
  atomicAdd(&c[1], cut);
  __syncthreads();
  if (threadIdx.x < 2) atomicMax(&most[threadIdx.x], c[threadIdx.x]);
}

// Ascending bitonic sort of n (a power of two) items in shared memory.
template <typename T>
__device__ void sort_shared(T* a, int n) {
  for (int k = 2; k <= n; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < n / 2; t += kTileBlock) {
        const int i = 2 * t - (t & (j - 1)), p = i + j;
        const T x = a[i], y = a[p];
        if ((x > y) == ((i & k) == 0)) {
          a[i] = y;
          a[p] = x;
        }
      }
    }
  __syncthreads();
}

// First index of a sorted list not below x.
template <typename T>
__device__ __forceinline__ int lower_bound(const T* a, int n, T x) {
  int lo = 0;
  while (n > 0) {
    const int h = n / 2;
    if (a[lo + h] < x) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo;
}

// The cells of each tile by device index: its rows of neighbouring cells are
// then neighbours in memory and in the block's shared memory.
__global__ void __launch_bounds__(kTileBlock) k_tile_sort(int32_t* order, int C, int T) {
  __shared__ int a[kTileMaxOwn];
  const int p0 = blockIdx.x * T, n = min(T, C - p0);
  for (int l = threadIdx.x; l < kTileMaxOwn; l += kTileBlock)
    a[l] = l < n ? order[p0 + l] : 0x7fffffff;
  sort_shared(a, kTileMaxOwn);
  for (int l = threadIdx.x; l < n; l += kTileBlock) order[p0 + l] = a[l];
}

// One block per tile. Faces by (boundary, branch bits, face), so that a warp
// of the flux phase takes one branch; halo cells by index.
__global__ void __launch_bounds__(kTileBlock) k_tile_build(const TileSource s, const TileArgs t,
                                                           int nf2, int nh2) {
  extern __shared__ __align__(16) unsigned char raw[];
  uint64_t* key = reinterpret_cast<uint64_t*>(raw);
  int* halo = reinterpret_cast<int*>(key + nf2);
  __shared__ int n_face, n_cut, n_halo;
  const int tile = blockIdx.x, tid = threadIdx.x;
  const int own = min(s.T, s.C - tile * s.T);
  if (tid == 0) n_face = n_cut = n_halo = 0;
  for (int i = tid; i < nf2; i += kTileBlock) key[i] = ~0ull;
  for (int i = tid; i < nh2; i += kTileBlock) halo[i] = 0x7fffffff;
  __syncthreads();
  auto face_key = [&](int f) {
    return (uint64_t)(f >= s.Fi) << 62 | (uint64_t)s.side[f] << 32 | (uint32_t)f;
  };
  for (int l = tid; l < own; l += kTileBlock)
    for_faces(s, tile, s.order[tile * s.T + l], [&](int, int f, int, int other, bool mine) {
      if (mine) key[atomicAdd(&n_face, 1)] = face_key(f);
      if (other >= 0 && s.pos[other] / s.T != tile) halo[atomicAdd(&n_cut, 1)] = other;
    });
  sort_shared(key, nf2);
  sort_shared(halo, nh2);
  // the halo cells once each, packed in place: all repeats to the end, sorted again
  const int ncut = n_cut;
  bool repeat[8];
  for (int i = tid, j = 0; i < ncut; i += kTileBlock, j++) repeat[j & 7] = i > 0 && halo[i] == halo[i - 1];
  __syncthreads();
  for (int i = tid, j = 0; i < ncut; i += kTileBlock, j++) {
    if (repeat[j & 7])
      halo[i] = 0x7fffffff;
    else
      atomicAdd(&n_halo, 1);
  }
  sort_shared(halo, nh2);
  const int nh = n_halo, nf = n_face;
  auto local = [&](int c) {
    const int p = s.pos[c];
    return p / s.T == tile ? p % s.T : own + lower_bound(halo, nh, c);
  };
  const size_t cb = (size_t)tile * t.SC, fb = (size_t)tile * t.SF;
  for (int l = tid; l < t.SC; l += kTileBlock) {
    const int c = l < own ? s.order[tile * s.T + l] : l < own + nh ? halo[l - own] : -1;
    t.cell[cb + l] = c;
    if (t.wset) t.wset[cb + l] = c >= 0 ? s.cell_wset[c] : 0;
    for (int k = 0; k < s.K; k++)
      t.nbr[((size_t)tile * s.K + k) * t.SC + l] = c >= 0 ? s.st_nbr[(size_t)k * s.C + c] : -1;
  }
  for (int i = tid; i < t.SF; i += kTileBlock) {
    uint32_t ij = 0;
    int fid = 0, rec = 0;
    if (i < nf) {
      const int f = (int)(uint32_t)(key[i] & 0xffffffffu), sd = (int)(key[i] >> 32 & 0x3fff);
      const int2 id = s.face_ids[f];
      const int ln = id.y < s.C ? local(id.y) : kTileGhost;
      ij = (uint32_t)local(id.x) | (uint32_t)ln << 11 | (uint32_t)(sd & 0x3ff) << 22;
      fid = (int)((uint32_t)f | (uint32_t)(sd >> 10) << 28);
      if (t.rec) rec = s.face_rec[f];
    }
    t.ij[fb + i] = ij;
    t.fid[fb + i] = fid;
    if (t.rec) t.rec[fb + i] = rec;
  }
  for (int l = tid; l < s.T; l += kTileBlock) {
    for (int k = 0; k < s.K2; k++) t.slot[((size_t)tile * s.K2 + k) * s.T + l] = 0xffff;
    if (l < own)
      for_faces(s, tile, s.order[tile * s.T + l], [&](int k, int f, int nb, int, bool) {
        t.slot[((size_t)tile * s.K2 + k) * s.T + l] =
            (uint16_t)(lower_bound(key, nf, face_key(f)) << 1 | nb);
      });
  }
  if (tid == 0) t.count[tile] = make_int2(own + nh, nf);
}

inline int grid_of(long long n) {
  const long long b = (n + kTileBlock - 1) / kTileBlock;
  return (int)(b < 4096 ? b : 4096);
}

inline int pow2_at_least(int n) {
  int p = 32;
  while (p < n) p <<= 1;
  return p;
}

}  // namespace

int hilbert_bits() { return 10; }

void launch_cell_curve(int C, const double* ccen, const double* vol, const int32_t* cell_new,
                       const CurveScratch& s, int32_t* order, cudaStream_t st) {
  const int bits = hilbert_bits();
  const int nblk = (C + kSortItems - 1) / kSortItems, n = 256 * nblk;
  k_bounds<<<kBoundsBlocks, kTileBlock, 0, st>>>(C, ccen, vol, s.part);
  k_box<<<1, 1, 0, st>>>(s.part, C, bits, s.part + 7 * kBoundsBlocks);
  k_hilbert<<<grid_of(C), kTileBlock, 0, st>>>(C, ccen, cell_new, s.part + 7 * kBoundsBlocks, bits,
                                               s.key[0], s.val[0]);
  int src = 0;
  for (int shift = 0; shift < 3 * bits; shift += 8, src ^= 1) {
    k_digit_count<<<nblk, kTileBlock, 0, st>>>(s.key[src], C, shift, nblk, s.count);
    launch_exclusive_scan(s.count, n, s.off, s.wsum, s.wbase, s.info, st);
    k_digit_place<<<nblk, kTileBlock, 0, st>>>(s.key[src], s.val[src], C, shift, nblk, s.off,
                                               s.wbase, s.key[src ^ 1], s.val[src ^ 1]);
  }
  cudaMemcpyAsync(order, s.val[src], 4 * (size_t)C, cudaMemcpyDeviceToDevice, st);
}

void launch_tile_order(int C, int T, int32_t* order, int32_t* pos, cudaStream_t st) {
  k_tile_sort<<<(C + T - 1) / T, kTileBlock, 0, st>>>(order, C, T);
  k_positions<<<grid_of(C), kTileBlock, 0, st>>>(order, C, pos);
}

CurveSizes curve_sizes(int C) {
  const size_t n = 256 * ((size_t)(C + kSortItems - 1) / kSortItems);
  return {7 * kBoundsBlocks + 4, n, (n + kFaceWindow - 1) / kFaceWindow};
}

void launch_face_sides(const KernelArgs& a, int precision, uint16_t* side, cudaStream_t st) {
  if (precision == PLFBS_FP32_DEVIATION)
    k_face_sides32<<<grid_of(a.F), kTileBlock, 0, st>>>(static_cast<const float4*>(a.face0),
                                                        static_cast<const float4*>(a.face1), a.F,
                                                        side);
  else if (a.flavour == PLFBS_FLAVOUR_CPU_SOLVER)
    k_face_sides<1><<<grid_of(a.F), kTileBlock, 0, st>>>(a.face0, a.face1, a.F, side);
  else
    k_face_sides<0><<<grid_of(a.F), kTileBlock, 0, st>>>(a.face0, a.face1, a.F, side);
}

static TileSource tile_source(const KernelArgs& a, const int32_t* order, const int32_t* pos,
                              const uint16_t* side, int T) {
  return TileSource{a.C,      a.F,      a.Fi,       a.K,         a.K2, T, order, pos,
                    reinterpret_cast<const int2*>(a.face_ids), a.gather, a.st_nbr, a.face_rec,
                    a.cell_wset, side};
}

void launch_tile_count(const KernelArgs& a, const int32_t* order, const int32_t* pos, int T,
                       int32_t* most, cudaStream_t st) {
  k_tile_count<<<(a.C + T - 1) / T, kTileBlock, 0, st>>>(tile_source(a, order, pos, nullptr, T),
                                                         most);
}

void launch_tile_build(const KernelArgs& a, const int32_t* order, const int32_t* pos,
                       const uint16_t* side, const TileArgs& t, int max_faces, int max_cut,
                       cudaStream_t st) {
  const int nf2 = pow2_at_least(max_faces), nh2 = pow2_at_least(max_cut);
  const size_t smem = 8 * (size_t)nf2 + 4 * (size_t)nh2;  // at most 40 KB (kTileMaxFaces, kTileMaxCells)
  k_tile_build<<<t.n, kTileBlock, smem, st>>>(tile_source(a, order, pos, side, t.T), t, nf2, nh2);
}

}  // namespace plfbs
