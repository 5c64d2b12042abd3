// FP64 record -> FP32 record, one edge a lane.
#pragma once

#include "vlm_bs.h"
#include "vlm_math.h"

namespace vlm {

// Lane k (0..3) of a record's four writes corner k and edge k of the FP32 record
// o (null: a lane without a record, which still takes part in the shuffles).
// p: the FP64 corner (of a single filament, end 1 in lanes 1 and 2, end 0 in
// lanes 0 and 3); rv: filament k's core radius.  The edge vectors are differenced
// in FP64 (nearby corners cancel) and rounded once; everything else is FP32.
// With edge weights (lattice form) edge k carries w and is active iff w != 0;
// without, every filament of a record carries its gam unless the record is
// skipped (|gam| <= eps with REC_SKIP), a single filament only its first.
// Inactive edges 2 and 3 are marked for the kernel to skip.
__device__ __forceinline__ void pack_edge32(d3 p, double rv, double g, int flags, bool weighted, double w, int k,
                                            float nf, float* __restrict__ o) {
  const int next = (threadIdx.x & 28) | ((k + 1) & 3);
  const double qx = __shfl_sync(0xffffffffu, p.x, next), qy = __shfl_sync(0xffffffffu, p.y, next),
               qz = __shfl_sync(0xffffffffu, p.z, next);
  if (!o) return;
  const bool skipped = (flags & REC_SKIP) && !(fabs(g) > kEps);
  const bool act = weighted ? w != 0.0 : (!(flags & REC_FIL) || k == 0) && !skipped;
  const float ex = (float)(qx - p.x), ey = (float)(qy - p.y), ez = (float)(qz - p.z);
  const float ee = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
  const float sk = (float)rv * sqrtf(ee);
  const float s2 = sk * sk;
  o[3 * k] = (float)p.x;
  o[3 * k + 1] = (float)p.y;
  o[3 * k + 2] = (float)p.z;
  const float wk = act ? (float)((weighted ? w : g) * kInv4Pi) : 0.f;
  o[12 + 3 * k] = wk * ex;
  o[12 + 3 * k + 1] = wk * ey;
  o[12 + 3 * k + 2] = wk * ez;
  o[24 + k] = wk * ee;
  o[28 + k] = weighted && k >= 2 && !act ? -1.f : fmaxf(s2 * s2, 1e-36f);
  const float nfs = nf * sk;
  o[32 + k] = act && nf > 0.f ? nfs * nfs : -1.f;
}

}  // namespace vlm
