// Device access to a case's state: vectors, indices, the frame's panel records
// and the wake nodes in target order.
#pragma once

#include "vlm_math.h"
#include "vlm_solver.h"

namespace vlm {

__device__ __forceinline__ d3 ld3(const double* p) { return mk3(p[0], p[1], p[2]); }
__device__ __forceinline__ void st3(double* p, d3 v) {
  p[0] = v.x;
  p[1] = v.y;
  p[2] = v.z;
}
__device__ __forceinline__ size_t ringI(const Dims& d, int b, int i, int j) {
  return (size_t)b * d.NW * d.ns + i + (size_t)d.NW * j;
}
__device__ __forceinline__ size_t velI(const Dims& d, int b, int i, int j) {
  return (size_t)b * d.NW * (d.ns + 1) + i + (size_t)d.NW * j;
}
__device__ __forceinline__ const double* panRec(const Dims& d, const double* fr, int b, int p) {
  return fr + d.fl.pan + ((size_t)b * d.npan + p) * kPan;
}

// Wake node m in target order: blade b, near-wake node (i, j) or far-wake filament i
constexpr int kTileRows = 16, kTileCols = 4;
__device__ __forceinline__ void decode_node(const Dims& d, int rowNear, int rowFar, int m, int& b, int& far, int& i,
                                            int& j) {
  const int rowsN = d.NW - (rowNear - 1);
  const int rowsF = max(d.NF - (rowFar - 1), 0);
  const int per = rowsN * (d.ns + 1) + rowsF;
  b = m / per;
  const int l = m % per;
  if (l < rowsN * (d.ns + 1)) {
    // tiles of kTileRows rows x kTileCols span stations, tile by tile: a run
    // of 32 consecutive targets (one warp's lanes in the FP32 kernel) is a
    // compact patch of the wake sheet, so few source rings come near any of
    // them
    far = 0;
    const int band = l / (kTileRows * (d.ns + 1));
    const int br = min(kTileRows, rowsN - band * kTileRows);
    const int o = l - band * kTileRows * (d.ns + 1);
    const int tc = o / (br * kTileCols);
    const int q = o - tc * br * kTileCols;
    i = rowNear - 1 + band * kTileRows + q % br;
    j = tc * kTileCols + q / br;
  } else {
    far = 1;
    j = 0;
    i = rowFar - 1 + (l - rowsN * (d.ns + 1));
  }
}

__device__ __forceinline__ d3 node_position(const Dims& d, const DevState& s, int rowNear, int rowFar, int pred, int m) {
  int b, far, i, j;
  decode_node(d, rowNear, rowFar, m, b, far, i, j);
  const double* nc = pred ? s.nCP : s.nC;
  if (far) return ld3((pred ? s.fCP : s.fC) + ((size_t)b * d.NF + i) * 6);
  return j < d.ns ? ld3(nc + ringI(d, b, i, j) * 12 + 3) : ld3(nc + ringI(d, b, i, d.ns - 1) * 12 + 6);
}

}  // namespace vlm
