// When a mesh marches in one kernel (march.cu) and when it takes the step graph,
// host side. Times are us per step, march : graph, on 148 SMs.
//
// Where the records of the compact layout are read, the march takes every mesh
// whose tiles fit (up to about 68,000 FP64 or 142,000 FP32 hexahedra): from shared
// memory where they are few (uniform boxes: 13,824 cells FP64 31 : 59, 64,000 64 :
// 86, FP32 128,000 70 : 85), and beyond that from L2, where a table still leaves
// most of a stage's bytes out (boxes graded along one axis, 68 to 1,480 records:
// FP64 4,096 cells 26 : 55, 33,000 58 : 71, 58,000 76 : 82, the worst of 20 meshes 84 :
// 80; FP32 33,000 43 : 63, 112,000 77 : 80, the worst of 18 87 : 87).
//
// With a record per face and weights per cell a tile waits for them at every
// face, so a march takes about 16 + 0.0475 SF us (FP32 17 + 0.024 SF) for SF faces
// in the largest tile, and the graph 52 + 0.18 us (47 + 0.1) per thousand faces of
// the mesh. FP64: SF 960 59 : 70, 1,152 70 : 76, 1,216 83 : 76 and 88 : 74, 1,440 94 : 78;
// FP32: SF 1,344 59 : 61, 1,664 56 : 66, 1,760 62 : 71, 2,048 104 : 68. A largest tile far
// above the mesh's mean loses earlier (SF n / F: FP64 SF 928, 1.77, 69 : 65; FP32 SF
// 1,216, 1.37, 63 : 57 and 1,760, 1.37, 77 : 65), unless the tiles are small anyway.
#pragma once

namespace plfbs {

// Whether a tiling of F faces over `sms` tiles may pass march_wins, asked before
// the tiles are built: a seventh of the faces or more lie between two tiles,
// which both count them.
inline bool march_may_win(bool compact, bool fp32, int sms, int F) {
  return compact || F <= (long long)sms * (fp32 ? 1600 : 1000);
}

// n tiles of at most SF faces; compact: the kernel reads the compact layout's
// records and weight sets.
inline bool march_wins(bool compact, bool fp32, int n, int SF, int F) {
  if (compact) return true;
  if (SF > (fp32 ? 1792 : 1184)) return false;
  return SF <= (fp32 ? 1152 : 896) || 100LL * SF * n <= 136LL * F;
}

}  // namespace plfbs
