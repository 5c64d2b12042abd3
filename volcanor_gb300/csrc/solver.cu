// Time-step kernels of the FP64 free-wake solver: wake shedding, ageing,
// dissipation, predictor/corrector convection with lattice continuity,
// strain, rollup and truncation, AIC assembly and inversion, circulation
// solve and loads.  Compiled with -fmad=false: each kernel performs, per
// element, exactly the IEEE operations of the reference routine it restates.
#include <math.h>

#include <algorithm>
#include <atomic>

#include "launch.h"
#include "exact64.h"
#include "state_dev.h"
#include "vlm_math.h"
#include "vlm_solver.h"

namespace vlm {

namespace {

__device__ __forceinline__ m33 frameT(const Dims& d, const double* fr, int b) {
  const double* t = fr + d.fl.rot + 10 + 9 * (b - 1);
  m33 T;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) T.a[r][c] = t[3 * r + c];
  return T;
}

inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

// ---- shed (classdef.f90:4297-4325) ---------------------------------------
// the trailing-edge row (the leading edge's: k_wake_begin)
__global__ void k_shed(Dims d, DevState s, const double* fr, int rowNear) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nb * d.ns) return;
  const int b = t / d.ns, j = t % d.ns;
  const int p = (d.nc - 1) + d.nc * j;
  const double* w = panRec(d, fr, b, p);
  const int r = max(rowNear - 1, 1) - 1;
  double* c = s.nC + ringI(d, b, r, j) * 12;
  st3(c + 3, ld3(w + 3));
  st3(c + 6, ld3(w + 6));
}

// ---- start of a step: the leading-edge row shed (classdef.f90:4297-4325), age
// (:4331-4354) and dissipation (:4356-4408), a ring or far filament a thread.
// A ring's third edge takes the new core radius of the row before: that row's
// thread writes it.  (Four kernels, 9 us of a hover step, now 4.)
__global__ void k_wake_begin(Dims d, DevState s, const double* fr, int rowNear, int rowFar, int dissip) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = d.nb * rows * d.ns;
  const int nFar = d.nb * max(d.NF - (rowFar - 1), 0);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nNear) {
    const int b = t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    const size_t r = ringI(d, b, i, j);
    double g = s.nGam[r];
    if (i == rowNear - 1) {
      const int p = (d.nc - 1) + d.nc * j;
      const double* w = panRec(d, fr, b, p);
      st3(s.nC + r * 12, ld3(w + 3));
      st3(s.nC + r * 12 + 9, ld3(w + 6));
      g = s.wGam[(size_t)b * d.npan + p];
    }
    s.nAge[r] = s.nAge[r] + d.dt;
    if (dissip) {
      double* rv = s.nRvc + 4 * r;
      const double c = sqrt(rv[0] * rv[0] + d.dissipAdd), e = sqrt(rv[1] * rv[1] + d.dissipAdd);
      rv[0] = c;
      rv[2] = c;
      rv[1] = e;
      if (i + 1 < d.NW) rv[4 + 3] = e;
      g = g * d.decay;
    }
    s.nGam[r] = g;
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int rf = d.NF - (rowFar - 1);
    const int b = l / rf, i = rowFar - 1 + l % rf;
    const size_t r = (size_t)b * d.NF + i;
    s.fAge[r] = s.fAge[r] + d.dt;
    if (dissip) {
      s.fRvc[r] = sqrt(s.fRvc[r] * s.fRvc[r] + d.dissipAdd);
      s.fGam[r] = s.fGam[r] * d.decay;
    }
  }
}

// ---- predictor and corrector ------------------------------------------------
// Convection moves corner 1 of every ring (and corner 2 of a row's last) by its
// node's velocity and then copies the corners that neighbours share
// (classdef.f90:1515-1575, 1609-1702).  These kernels form a ring's or filament's
// new corners from the old ones of itself and its neighbours and write them
// elsewhere, so that one pass does what the copy, the shift and the continuity
// did one after the other.
// node (i, j) after convection; the predicted wake moves row 1 alone
__device__ __forceinline__ d3 moved_node(const Dims& d, const DevState& s, int b, int i, int j, bool moves) {
  const d3 p = j < d.ns ? ld3(s.nC + ringI(d, b, i, j) * 12 + 3) : ld3(s.nC + ringI(d, b, i, d.ns - 1) * 12 + 6);
  return moves ? p + ld3(s.vN[0] + 3 * velI(d, b, i, j)) * d.dt : p;
}
struct Ring4 {
  d3 c0, c1, c2, c3;
};
__device__ __forceinline__ Ring4 convected(const Dims& d, const DevState& s, int b, int i, int j, int rowNear, bool pred) {
  Ring4 o;
  const double* c = s.nC + ringI(d, b, i, j) * 12;
  const bool moves = !pred || i == 0, above = !pred || i - 1 == 0;
  o.c1 = moved_node(d, s, b, i, j, moves);
  o.c2 = moved_node(d, s, b, i, j + 1, moves);
  if (i > rowNear - 1) {
    o.c0 = moved_node(d, s, b, i - 1, j, above);
    o.c3 = moved_node(d, s, b, i - 1, j + 1, above);
  } else {
    o.c0 = ld3(c);
    o.c3 = ld3(c + 9);
  }
  return o;
}
// a far filament's ends after convection: the second is its predecessor's first
__device__ __forceinline__ void convected_far(const Dims& d, const DevState& s, int b, int i, int rowFar, d3& a, d3& e) {
  const size_t f = (size_t)b * d.NF + i;
  a = ld3(s.fC + 6 * f) + ld3(s.vF[0] + 3 * f) * d.dt;
  e = i > rowFar - 1 ? ld3(s.fC + 6 * (f - 1)) + ld3(s.vF[0] + 3 * (f - 1)) * d.dt : ld3(s.fC + 6 * f + 3);
}
__device__ __forceinline__ void put_ring(double* c, const Ring4& r) {
  st3(c, r.c0);
  st3(c + 3, r.c1);
  st3(c + 6, r.c2);
  st3(c + 9, r.c3);
}

// The predicted wake (main.f90:1012-1019 and its convection).  (Copy, shift and
// continuity: 10 us of a hover step, now 3.4.)
__global__ void k_predict(Dims d, DevState s, int rowNear, int rowFar) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = d.nb * rows * d.ns;
  const int nFar = d.nb * max(d.NF - (rowFar - 1), 0);
  const int nRow1 = rowNear > 1 ? d.nb * d.ns : 0;  // row 1 moves even where it is not in use
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nNear) {
    const int b = t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    put_ring(s.nCP + ringI(d, b, i, j) * 12, convected(d, s, b, i, j, rowNear, true));
    return;
  }
  t -= nNear;
  if (t < nFar) {
    const int rf = d.NF - (rowFar - 1);
    const int b = t / rf, i = rowFar - 1 + t % rf;
    d3 a, e;
    convected_far(d, s, b, i, rowFar, a, e);
    double* c = s.fCP + ((size_t)b * d.NF + i) * 6;
    st3(c, a);
    st3(c + 3, e);
    return;
  }
  t -= nFar;
  if (t < nRow1) {
    const int b = t / d.ns, j = t % d.ns;
    double* c = s.nCP + ringI(d, b, 0, j) * 12;
    st3(c + 3, ld3(c + 3) + ld3(s.vN[0] + 3 * velI(d, b, 0, j)) * d.dt);
    if (j == d.ns - 1) st3(c + 6, ld3(c + 6) + ld3(s.vN[0] + 3 * velI(d, b, 0, d.ns)) * d.dt);
  }
}

// The corrector's convection, out of place, with the far wake's strain
// (classdef.f90:4410-4422, 505-521): rings into nTmp (18 doubles: corners,
// circulation, core radii, age), far filaments into fTmp (12).
__global__ void k_correct(Dims d, DevState s, int rowNear, int rowFar, int strain) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = d.nb * rows * d.ns;
  const int nFar = d.nb * max(d.NF - (rowFar - 1), 0);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nNear) {
    const int b = t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    const size_t r = ringI(d, b, i, j);
    double* o = s.nTmp + r * 18;
    put_ring(o, convected(d, s, b, i, j, rowNear, false));
    o[12] = s.nGam[r];
    for (int k = 0; k < 4; ++k) o[13 + k] = s.nRvc[4 * r + k];
    o[17] = s.nAge[r];
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int rf = d.NF - (rowFar - 1);
    const int b = l / rf, i = rowFar - 1 + l % rf;
    const size_t f = (size_t)b * d.NF + i;
    double* o = s.fTmp + f * 12;
    d3 a, e;
    convected_far(d, s, b, i, rowFar, a, e);
    st3(o, a);
    st3(o + 3, e);
    double rv = s.fRvc[f], lc = s.fLc[f];
    if (strain) {
      lc = norm3(a - e);
      rv = s.fRvc0[f] * sqrt(s.fL0[f] / lc);
    }
    o[6] = s.fGam[f];
    o[7] = rv;
    o[8] = s.fRvc0[f];
    o[9] = s.fL0[f];
    o[10] = lc;
    o[11] = s.fAge[f];
  }
}

__device__ __forceinline__ void velop(const DevState& s, bool nearPart, long e, int op);

// Back into the state: with row 1 in use the last row is rolled up into the far
// wake (classdef.f90:4515-4605) and every row moves on by one (:4481-4498), the far
// wake too when it is full (:4500-4513); the trailing-edge row is shed; the
// velocity history moves on.  The rollup has a warp per blade: a lane for each
// sum (the leading and trailing corner's components, the circulation, the core
// radius), so that only the additions of one are serial.  (Convection, velocity
// algebra, rollup, row moves and shedding in ten kernels: 36 us of a hover
// step, now 10.)
__global__ void k_correct_back(Dims d, DevState s, const double* fr, int rowNear, int rowFar, int op, int rollBlocks) {
  after_previous();
  const bool roll = rowNear == 1, full = roll && d.NF > 0 && rowFar == 1;
  const int rowNext = full ? 1 : rowFar - 1;  // the far row that the rollup fills
  if ((int)blockIdx.x < rollBlocks) {
    const int lane = threadIdx.x & 31, b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= d.nb) return;
    auto ring = [&](int j) { return s.nTmp + ringI(d, b, d.NW - 1, j) * 18; };
    double gamRollup = ring(d.ns - 1)[12];
    const bool posSense = fsign1(d.omega * d.theta0) > kEps;
    double sum = 0.0;
    const int c = lane < 3 ? 9 + lane : lane < 6 ? 3 + lane : lane == 6 ? 12 : 15;  // of the ring's 18
#pragma unroll 4
    for (int is = d.rollupStart; is <= d.rollupEnd; ++is) {
      const double* q = ring(is - 1);
      const double g = q[12], x = q[c];
      sum = lane == 6 ? sum + g : sum + x * g;
      if (posSense ? g < gamRollup : g > gamRollup) gamRollup = g;
    }
    const double gamSum = __shfl_sync(0xffffffffu, sum, 6);
    if (fabs(gamSum) > kEps) {
      sum = sum / gamSum;
    } else {
      const double* q = ring(d.rollupEnd - 1);
      sum = lane < 3 ? q[3 + lane] : lane < 6 ? q[3 + lane] : q[15];
    }
    const double x = __shfl_sync(0xffffffffu, sum, lane < 3 ? lane + 3 : lane);  // cTE
    const double df = x - sum;                                                   // cTE - cLE, lanes 0 to 2
    const d3 dv = mk3(__shfl_sync(0xffffffffu, df, 0), __shfl_sync(0xffffffffu, df, 1), __shfl_sync(0xffffffffu, df, 2));
    if (d.suppressFwake == 1) gamRollup = 0.0;
    const size_t f = (size_t)b * d.NF + (rowNext - 1);
    if (lane < 3) {
      s.fC[6 * f + 3 + lane] = sum;
      s.fC[6 * f + lane] = x;
      if (rowNext < d.NF) s.fC[6 * (f + 1) + 3 + lane] = x;
    }
    if (lane == 7) {
      s.fGam[f] = gamRollup;
      s.fAge[f] = ring(d.ns - 1)[17];
      s.fRvc0[f] = sum;
      s.fRvc[f] = sum;
      const double lc = norm3(dv);
      s.fLc[f] = lc;
      s.fL0[f] = lc;
    }
    return;
  }
  long t = (long)(blockIdx.x - rollBlocks) * blockDim.x + threadIdx.x;
  const int rows = d.NW - (rowNear - 1), nNear = d.nb * rows * d.ns;
  if (t < nNear) {
    const int b = (int)t / (rows * d.ns), l = (int)t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    const size_t r = ringI(d, b, i, j);
    const double* o = s.nTmp + (roll && i > 0 ? r - 1 : r) * 18;
    double* c = s.nC + 12 * r;
    const double* w = roll && i == 0 ? panRec(d, fr, b, (d.nc - 1) + d.nc * j) : nullptr;  // the shed row's trailing edge
    st3(c, ld3(o));
    st3(c + 3, ld3(w ? w + 3 : o + 3));
    st3(c + 6, ld3(w ? w + 6 : o + 6));
    st3(c + 9, ld3(o + 9));
    if (roll) {
      s.nGam[r] = o[12];
      for (int k = 0; k < 4; ++k) s.nRvc[4 * r + k] = o[13 + k];
      s.nAge[r] = i == 0 ? 0.0 : o[17];
    }
    return;
  }
  t -= nNear;
  const int rf = max(d.NF - (rowFar - 1), 0), nFar = d.nb * rf;
  if (t < nFar) {
    const int b = (int)t / rf, i = rowFar - 1 + (int)t % rf;
    const size_t f = (size_t)b * d.NF + i;
    if (full && i == 0) return;  // the rollup's
    const double* o = s.fTmp + (full ? f - 1 : f) * 12;
    st3(s.fC + 6 * f, ld3(o));
    if (!(roll && i == rowNext)) st3(s.fC + 6 * f + 3, ld3(o + 3));  // row rowNext + 1's second end is the rollup's
    s.fGam[f] = o[6];
    s.fRvc[f] = o[7];
    s.fRvc0[f] = o[8];
    s.fL0[f] = o[9];
    s.fLc[f] = o[10];
    s.fAge[f] = o[11];
    return;
  }
  t -= nFar;
  const int nShed = roll ? 0 : d.nb * d.ns;
  if (t < nShed) {
    const int b = (int)t / d.ns, j = (int)t % d.ns;
    const double* w = panRec(d, fr, b, (d.nc - 1) + d.nc * j);
    double* c = s.nC + ringI(d, b, rowNear - 2, j) * 12;
    st3(c + 3, ld3(w + 3));
    st3(c + 6, ld3(w + 6));
    return;
  }
  t -= nShed;
  const long nN = (long)d.nb * d.NW * (d.ns + 1) * 3, nF = (long)d.nb * d.NF * 3;
  if (op >= 0 && t < nN + nF) velop(s, t < nN, t < nN ? t : t - nN, op);
}

// ---- predicted copy (main.f90:1012-1019) -----------------------------------
__global__ void k_copy_pred(Dims d, DevState s, int rowNear, int rowFar) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = d.nbC * rows * d.ns;
  const int nFar = d.nbC * max(d.NF - (rowFar - 1), 0);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nNear) {
    const int b = t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    const size_t r = ringI(d, b, i, j) * 12;
    for (int k = 0; k < 12; ++k) s.nCP[r + k] = s.nC[r + k];
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int rf = d.NF - (rowFar - 1);
    const int b = l / rf, i = rowFar - 1 + l % rf;
    const size_t r = ((size_t)b * d.NF + i) * 6;
    for (int k = 0; k < 6; ++k) s.fCP[r + k] = s.fC[r + k];
  }
}

// ---- convection shift (classdef.f90:1515-1575) ----------------------------
__global__ void k_shift(Dims d, DevState s, int rowNear, int rowFar, int pred) {
  after_previous();
  const int rows = pred ? 1 : d.NW - (rowNear - 1);
  const int i0 = pred ? 0 : rowNear - 1;  // the predicted loop visits row 1 only
  const int nNear = d.nbC * rows * (d.ns + 1);
  const int nFar = d.nbC * max(d.NF - (rowFar - 1), 0);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double* nc = pred ? s.nCP : s.nC;
  if (t < nNear) {
    const int b = t / (rows * (d.ns + 1)), l = t % (rows * (d.ns + 1));
    const int j = l / rows, i = i0 + l % rows;
    const d3 dv = ld3(s.vN[0] + 3 * velI(d, b, i, j)) * d.dt;
    double* c = j < d.ns ? nc + ringI(d, b, i, j) * 12 + 3 : nc + ringI(d, b, i, d.ns - 1) * 12 + 6;
    st3(c, ld3(c) + dv);
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int rf = d.NF - (rowFar - 1);
    const int b = l / rf, i = rowFar - 1 + l % rf;
    double* c = (pred ? s.fCP : s.fC) + ((size_t)b * d.NF + i) * 6;
    st3(c, ld3(c) + ld3(s.vF[0] + 3 * ((size_t)b * d.NF + i)) * d.dt);
  }
}

// ---- continuity (classdef.f90:1609-1702) ----------------------------------
__global__ void k_continuity(Dims d, DevState s, int rowNear, int rowFar, int pred) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = d.nbC * rows * d.ns;
  const int nFar = d.nbC * max(d.NF - rowFar, 0);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double* nc = pred ? s.nCP : s.nC;
  if (t < nNear) {
    const int b = t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    double* c = nc + ringI(d, b, i, j) * 12;
    if (i > rowNear - 1) {
      if (j < d.ns - 1) {
        st3(c + 0, ld3(nc + ringI(d, b, i - 1, j) * 12 + 3));
        st3(c + 6, ld3(nc + ringI(d, b, i, j + 1) * 12 + 3));
        st3(c + 9, ld3(nc + ringI(d, b, i - 1, j + 1) * 12 + 3));
      } else {
        st3(c + 0, ld3(nc + ringI(d, b, i - 1, j) * 12 + 3));
        st3(c + 9, ld3(nc + ringI(d, b, i - 1, j) * 12 + 6));
      }
    } else if (j < d.ns - 1) {
      st3(c + 6, ld3(nc + ringI(d, b, i, j + 1) * 12 + 3));
    }
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int rf = d.NF - rowFar;
    const int b = l / rf, i = rowFar + l % rf;
    double* fc = pred ? s.fCP : s.fC;
    st3(fc + ((size_t)b * d.NF + i) * 6 + 3, ld3(fc + ((size_t)b * d.NF + i - 1) * 6));
  }
}

// ---- axisymmetric wake copies (classdef.f90:4801-4823) ---------------------
__global__ void k_axisym(Dims d, DevState s, const double* fr, int rowNear, int rowFar, int pred) {
  after_previous();
  const int rows = d.NW - (rowNear - 1);
  const int nNear = (d.nb - 1) * rows * d.ns;
  const int rf = max(d.NF - (rowFar - 1), 0);
  const int nFar = (d.nb - 1) * rf;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const d3 hub = ld3(fr + d.fl.rot + 3);
  if (t < nNear) {
    const int b = 1 + t / (rows * d.ns), l = t % (rows * d.ns);
    const int j = l / rows, i = rowNear - 1 + l % rows;
    const m33 T = frameT(d, fr, b);
    const size_t r0 = ringI(d, 0, i, j), r1 = ringI(d, b, i, j);
    double* nc = pred ? s.nCP : s.nC;
    for (int k = 0; k < 4; ++k) st3(nc + r1 * 12 + 3 * k, rot_about(T, ld3(nc + r0 * 12 + 3 * k), hub));
    if (!pred) {
      s.nGam[r1] = s.nGam[r0];
      for (int k = 0; k < 4; ++k) s.nRvc[4 * r1 + k] = s.nRvc[4 * r0 + k];
      s.nAge[r1] = s.nAge[r0];
    }
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int b = 1 + l / rf, i = rowFar - 1 + l % rf;
    const m33 T = frameT(d, fr, b);
    const size_t r0 = i, r1 = (size_t)b * d.NF + i;
    double* fc = pred ? s.fCP : s.fC;
    st3(fc + r1 * 6, rot_about(T, ld3(fc + r0 * 6), hub));
    st3(fc + r1 * 6 + 3, rot_about(T, ld3(fc + r0 * 6 + 3), hub));
    if (!pred) {
      s.fGam[r1] = s.fGam[r0];
      s.fRvc[r1] = s.fRvc[r0];
      s.fRvc0[r1] = s.fRvc0[r0];
      s.fL0[r1] = s.fL0[r0];
      s.fLc[r1] = s.fLc[r0];
      s.fAge[r1] = s.fAge[r0];
    }
  }
}

// ---- strain (classdef.f90:4410-4422, 505-521) ------------------------------
__global__ void k_strain(Dims d, DevState s, int rowFar) {
  after_previous();
  const int rf = d.NF - (rowFar - 1);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (rf <= 0 || t >= d.nb * rf) return;
  const int b = t / rf, i = rowFar - 1 + t % rf;
  const size_t r = (size_t)b * d.NF + i;
  const double lc = norm3(ld3(s.fC + 6 * r) - ld3(s.fC + 6 * r + 3));
  s.fLc[r] = lc;
  s.fRvc[r] = s.fRvc0[r] * sqrt(s.fL0[r] / lc);
}

// ---- prescribed far wake (classdef.f90:998-1066, 5172-5217) ----------------
// One block per convecting blade.  Thread 0 sums the far-wake filaments
// rowStart..NF in the reference's order (radius of node 1 about the z axis,
// descent between consecutive nodes), relaxes the helix pitch and radius,
// and finds the anchor (node 1 of the oldest filament); the threads then
// place the 241 helix nodes about the hub, filament i running from node i+1
// to node i, the first one attached at the anchor.  The helix angles use
// the device's cos/sin/atan2, so the nodes agree with a host evaluation to a
// few ulps, not bit for bit.
__global__ void k_presc_update(Dims d, DevState s, const double* fr, int rowFar, int pred) {
  after_previous();
  const int b = blockIdx.x;
  const int rowStart = d.prescGenNt == 0 ? rowFar : d.NF - d.prescGenNt;
  const int i0 = rowStart - 1, i1 = d.NF - 1, n = i1 - i0 + 1;
  const double* fc = (pred ? s.fCP : s.fC) + (size_t)b * d.NF * 6;
  double* H = s.pfHelix + 2 * ((size_t)pred * d.nb + b);
  __shared__ double sh[6];  // pitch, radius, anchor xyz, dTheta
  if (threadIdx.x == 0) {
    double pitch = 0.0, radius = 0.0;
    for (int i = 0; i < n; ++i) {
      const double* c = fc + 6 * (size_t)(i0 + i);
      radius = radius + sqrt(c[1] * c[1] + c[0] * c[0]);
      if (i < n - 1) pitch = pitch + c[2] - fc[6 * (size_t)(i0 + i + 1) + 2];
    }
    const double dpsi = fr[d.fl.rot + 9] * d.dt;
    pitch = fabs(pitch) * (-kTwoPi / dpsi) / (double)(n - 1);
    radius = radius / (double)n;
    H[0] = 0.5 * pitch + (1.0 - 0.5) * H[0];
    H[1] = 0.5 * radius + (1.0 - 0.5) * H[1];
    const double* a = fc + 6 * (size_t)i1;
    sh[0] = H[0];
    sh[1] = H[1];
    sh[2] = a[0], sh[3] = a[1], sh[4] = a[2];
    sh[5] = atan2(a[1], a[0]);
    s.pfGam[(size_t)pred * d.nb + b] = (pred ? s.fGam : s.fGam)[(size_t)b * d.NF + i1];
    s.pfRvc[(size_t)pred * d.nb + b] = s.fRvc[(size_t)b * d.NF + i1];
  }
  __syncthreads();
  __shared__ double node[3 * (kPresc + 1)];
  const d3 hub = ld3(fr + d.fl.rot + 3);
  const double dx = (kTwoPi * 10.0 - 0.0) / (double)kPresc;  // linspace(0, 2 pi nRevs, 241)
  for (int i = threadIdx.x; i <= kPresc; i += blockDim.x) {
    const double th = -1.0 * ((double)i * dx + 0.0);  // a clockwise helix (isClockwiseRotor)
    node[3 * i] = hub.x + sh[1] * cos(th + sh[5]);
    node[3 * i + 1] = hub.y + sh[1] * sin(th + sh[5]);
    node[3 * i + 2] = hub.z + (sh[0] * fabs(th) / kTwoPi + (sh[4] - hub.z));
  }
  __syncthreads();
  double* out = s.pfC + ((size_t)pred * d.nb + b) * kPresc * 6;
  for (int i = threadIdx.x; i < kPresc; i += blockDim.x) {
    for (int k = 0; k < 3; ++k) out[6 * i + k] = node[3 * (i + 1) + k];  // fc1
    for (int k = 0; k < 3; ++k) out[6 * i + 3 + k] = i == 0 ? sh[2 + k] : node[3 * i + k];  // fc2
  }
}
// Axisymmetric copies: blade b's prescribed wake = blade 1's, rotated about
// the hub by b x 2 pi / nb (the wake copies' rotation).
__global__ void k_presc_axisym(Dims d, DevState s, const double* fr, int pred) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (d.nb - 1) * kPresc) return;
  const int b = 1 + t / kPresc, i = t % kPresc;
  const m33 T = frameT(d, fr, b);
  const d3 hub = ld3(fr + d.fl.rot + 3);
  const double* src = s.pfC + ((size_t)pred * d.nb) * kPresc * 6 + 6 * (size_t)i;
  double* dst = s.pfC + ((size_t)pred * d.nb + b) * kPresc * 6 + 6 * (size_t)i;
  st3(dst, rot_about(T, ld3(src), hub));
  st3(dst + 3, rot_about(T, ld3(src + 3), hub));
  if (i == 0) {
    s.pfGam[(size_t)pred * d.nb + b] = s.pfGam[(size_t)pred * d.nb];
    s.pfRvc[(size_t)pred * d.nb + b] = s.pfRvc[(size_t)pred * d.nb];
    s.pfHelix[2 * ((size_t)pred * d.nb + b)] = s.pfHelix[2 * (size_t)pred * d.nb];
    s.pfHelix[2 * ((size_t)pred * d.nb + b) + 1] = s.pfHelix[2 * (size_t)pred * d.nb + 1];
  }
}

// ---- wake burst (classdef.f90:4911-4917, 2306-2339) -------------------------
// Far-wake filament i of every blade against filament i+1: skew =
// |acos(cos(angle between fc2 - fc1 of i and fc1 - fc2 of i+1)) - pi| / pi;
// at or above skewLimit both get the chord as core radius.  Only core radii
// are written, from positions only, so the pairs run in parallel.
__global__ void k_burst(Dims d, DevState s, int rowFar) {
  after_previous();
  const int rf = d.NF - (rowFar - 1) - 1;  // pairs (i, i+1)
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (rf <= 0 || t >= d.nb * rf) return;
  const int b = t / rf, i = rowFar - 1 + t % rf;
  const size_t r = (size_t)b * d.NF + i;
  const d3 a = ld3(s.fC + 6 * r + 3) - ld3(s.fC + 6 * r);
  const d3 c = ld3(s.fC + 6 * (r + 1)) - ld3(s.fC + 6 * (r + 1) + 3);
  const double skew = fabs(acos(dot3(a, c) / sqrt(dot3(a, a) * dot3(c, c))) - kPi) / kPi;
  if (skew >= d.skewLimit) {
    s.fRvc[r + 1] = d.chord;
    s.fRvc[r] = d.chord;
  }
}

// ---- far-wake shift for truncation (classdef.f90:4500-4513) ----------------
__global__ void k_far_to_tmp(Dims d, DevState s) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nb * d.NF) return;
  const int b = t / d.NF, i = t % d.NF;
  const size_t src = (size_t)b * d.NF + (i > 0 ? i - 1 : 0);
  double* o = s.fTmp + (size_t)t * 12;
  for (int k = 0; k < 6; ++k) o[k] = s.fC[6 * src + k];
  o[6] = s.fGam[src];
  o[7] = s.fRvc[src];
  o[8] = s.fRvc0[src];
  o[9] = s.fL0[src];
  o[10] = s.fLc[src];
  o[11] = i == 0 ? 0.0 : s.fAge[src];
}
__global__ void k_far_from_tmp(Dims d, DevState s) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nb * d.NF) return;
  const double* o = s.fTmp + (size_t)t * 12;
  for (int k = 0; k < 6; ++k) s.fC[6 * (size_t)t + k] = o[k];
  s.fGam[t] = o[6];
  s.fRvc[t] = o[7];
  s.fRvc0[t] = o[8];
  s.fL0[t] = o[9];
  s.fLc[t] = o[10];
  s.fAge[t] = o[11];
}

// ---- rollup (classdef.f90:4515-4605) ---------------------------------------
__global__ void k_rollup(Dims d, DevState s, int rowFarNext) {
  after_previous();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= d.nb) return;
  const int NW = d.NW;
  auto ring = [&](int j) { return ringI(d, b, NW - 1, j); };
  double gamRollup = s.nGam[ring(d.ns - 1)];
  d3 cLE = zero3(), cTE = zero3();
  double radius = 0.0, gamSum = 0.0;
  const bool posSense = fsign1(d.omega * d.theta0) > kEps;
  for (int is = d.rollupStart; is <= d.rollupEnd; ++is) {
    const size_t r = ring(is - 1);
    const double g = s.nGam[r];
    cLE = cLE + ld3(s.nC + r * 12 + 9) * g;
    cTE = cTE + ld3(s.nC + r * 12 + 6) * g;
    gamSum = gamSum + g;
    if (posSense) {
      if (g < gamRollup) gamRollup = g;
    } else {
      if (g > gamRollup) gamRollup = g;
    }
    radius = radius + s.nRvc[4 * r + 2] * g;
  }
  const double ageRollup = s.nAge[ring(d.ns - 1)];
  if (fabs(gamSum) > kEps) {
    cLE = cLE / gamSum;
    cTE = cTE / gamSum;
    radius = radius / gamSum;
  } else {
    const size_t r = ring(d.rollupEnd - 1);
    cLE = ld3(s.nC + r * 12 + 3);
    cTE = ld3(s.nC + r * 12 + 6);
    radius = s.nRvc[4 * r + 2];
  }
  if (d.suppressFwake == 1) gamRollup = 0.0;
  if (d.NF > 0) {
    const size_t f = (size_t)b * d.NF + (rowFarNext - 1);
    st3(s.fC + 6 * f + 3, cLE);
    st3(s.fC + 6 * f, cTE);
    s.fGam[f] = gamRollup;
    s.fAge[f] = ageRollup;
    s.fRvc0[f] = radius;
    s.fRvc[f] = radius;
    const double lc = norm3(cTE - cLE);
    s.fLc[f] = lc;
    s.fL0[f] = lc;
    if (rowFarNext < d.NF) st3(s.fC + 6 * (f + 1) + 3, cTE);
  }
}

// ---- near-wake shift after rollup (classdef.f90:4481-4498) -----------------
__global__ void k_near_to_tmp(Dims d, DevState s) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int per = d.NW * d.ns;
  if (t >= d.nb * per) return;
  const int b = t / per, l = t % per;
  const int i = l % d.NW, j = l / d.NW;
  const size_t src = ringI(d, b, i > 0 ? i - 1 : 0, j);
  double* o = s.nTmp + (size_t)t * 18;
  for (int k = 0; k < 12; ++k) o[k] = s.nC[12 * src + k];
  o[12] = s.nGam[src];
  for (int k = 0; k < 4; ++k) o[13 + k] = s.nRvc[4 * src + k];
  o[17] = i == 0 ? 0.0 : s.nAge[src];
}
__global__ void k_near_from_tmp(Dims d, DevState s) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nb * d.NW * d.ns) return;
  const double* o = s.nTmp + (size_t)t * 18;
  for (int k = 0; k < 12; ++k) s.nC[12 * (size_t)t + k] = o[k];
  s.nGam[t] = o[12];
  for (int k = 0; k < 4; ++k) s.nRvc[4 * (size_t)t + k] = o[13 + k];
  s.nAge[t] = o[17];
}

// ---- velocity history algebra (main.f90:844-1406) --------------------------
__device__ __forceinline__ void velop(const DevState& s, bool nearPart, long e, int op) {
  double* a[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) a[k] = nearPart ? s.vN[k] : s.vF[k];
  double v = a[0][e], v1 = a[1][e], v2 = a[2][e], v3 = a[3][e], vp = a[4][e], st = a[5][e];
  switch (op) {
    case VOP_COPY_0_TO_1: a[1][e] = v; break;
    case VOP_COPY_0_TO_2: a[2][e] = v; break;
    case VOP_COPY_0_TO_3: a[3][e] = v; break;
    case VOP_AB2: {
      const double x = 0.5 * (3.0 * v - v1);
      a[5][e] = x;
      a[1][e] = x;
      a[0][e] = x;
    } break;
    case VOP_AM2_PRED:
      a[5][e] = v;
      a[0][e] = 0.5 * (3.0 * v - v1);
      break;
    case VOP_AM2_CORR: a[0][e] = (vp + st) * 0.5; break;
    case VOP_STEP_TO_1: a[1][e] = st; break;
    case VOP_AM3_PRED:
      a[5][e] = v;
      a[0][e] = ((23.0 * v - 16.0 * v2) + 5.0 * v1) / 12.0;
      break;
    case VOP_AM3_CORR: a[0][e] = ((5.0 * vp + 8.0 * st) - 1.0 * v2) / 12.0; break;
    case VOP_AM3_SHIFT:
      a[1][e] = v2;
      a[2][e] = st;
      break;
    case VOP_AM4_PRED:
      a[5][e] = v;
      a[0][e] = (((55.0 * v - 59.0 * v3) + 37.0 * v2) - 9.0 * v1) / 24.0;
      break;
    case VOP_AM4_CORR: a[0][e] = (((9.0 * vp + 19.0 * st) - 5.0 * v3) + 1.0 * v2) / 24.0; break;
    case VOP_AM4_SHIFT:
      a[1][e] = v2;
      a[2][e] = v3;
      a[3][e] = st;
      break;
  }
}
__global__ void k_velop(DevState s, long nN, long nF, int op) {
  after_previous();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t < nN + nF) velop(s, t < nN, t < nN ? t : t - nN, op);
}

// ---- PC2 averaging (libCommon.f90:213-258) ---------------------------------
__global__ void k_order2(Dims d, DevState s, int rowNear, int rowFar, int phase) {
  after_previous();
  const int m = d.NW - (rowNear - 1);
  const int mf = max(d.NF - (rowFar - 1), 0);
  const int nNear = d.nbC * (d.ns + 1) * m * 3;
  const int nFar = d.nbC * mf * 3;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nNear) {
    const int k = t % 3, q = t / 3;
    const int b = q / ((d.ns + 1) * m), l = q % ((d.ns + 1) * m);
    const int j = l / m, i = l % m;
    const size_t base = velI(d, b, rowNear - 1, j);
    const double* vn = s.vN[0] + 3 * base + k;
    const double* vp = s.vN[4] + 3 * base + k;
    double* tmp = s.vN[6] + 3 * base + k;
    if (phase == 0) {
      double o;
      if (i == 0) o = (vp[0] + vn[0]) * 0.5;
      else if (i < m - 1) o = (((vp[3 * i] + vp[3 * (i - 1)]) + vn[3 * (i + 1)]) + vn[3 * i]) * 0.25;
      else o = (vp[3 * i] + vn[3 * i]) * 0.5;
      if (i == m - 1) o = (vp[3 * i] + vn[3 * i]) * 0.5;
      tmp[3 * i] = o;
    } else {
      s.vN[0][3 * base + k + 3 * i] = tmp[3 * i];
    }
  } else if (t < nNear + nFar) {
    const int l = t - nNear;
    const int k = l % 3, q = l / 3;
    const int b = q / mf, i = q % mf;
    const size_t base = (size_t)b * d.NF + (rowFar - 1);
    const double* vn = s.vF[0] + 3 * base + k;
    const double* vp = s.vF[4] + 3 * base + k;
    double* tmp = s.vF[6] + 3 * base + k;
    if (phase == 0) {
      double o;
      if (i == 0) o = (vp[0] + vn[0]) * 0.5;
      else if (i < mf - 1) o = (((vp[3 * i] + vp[3 * (i - 1)]) + vn[3 * (i + 1)]) + vn[3 * i]) * 0.25;
      else o = (vp[3 * i] + vn[3 * i]) * 0.5;
      if (i == mf - 1) o = (vp[3 * i] + vn[3 * i]) * 0.5;
      tmp[3 * i] = o;
    } else {
      s.vF[0][3 * base + k + 3 * i] = tmp[3 * i];
    }
  }
}

__global__ void k_scatter_nodes(Dims d, DevState s, const double* fr, int rowNear, int rowFar, int pred,
                                double initWakeVel, int addInit, int op, int M) {
  after_previous();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  int b, far, i, j;
  decode_node(d, rowNear, rowFar, m, b, far, i, j);
  d3 v = ld3(s.outv + 3 * (size_t)m);
  if (addInit) {
    const d3 a = initWakeVel * ld3(fr + d.fl.rot + 6);
    if (pred || far) v = v - a;
    else v = v + a;
  }
  const size_t e = 3 * (far ? (size_t)b * d.NF + i : velI(d, b, i, j));
  st3((far ? s.vF : s.vN)[pred ? 4 : 0] + e, v);
  if (op >= 0)
    for (int c = 0; c < 3; ++c) velop(s, !far, (long)e + c, op);
}

// ---- AIC and its inverse (classdef.f90:4151-4179, libMath.f90:48-83) ---------
__global__ void k_aic(Dims d, DevState s, const double* fr) {
  after_previous();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long n = d.n;
  if (t >= n * n) return;
  const int row = (int)(t % n), col = (int)(t / n);
  const double* cp = panRec(d, fr, row / d.npan, row % d.npan);
  const double* w = panRec(d, fr, col / d.npan, col % d.npan);
  d3 c[4] = {ld3(w), ld3(w + 3), ld3(w + 6), ld3(w + 9)};
  const d3 v = exact64::vr_vind(exact64::load_unit(), ld3(cp + 12), c, s.wRvc + 4 * (size_t)col);
  s.AIC[row + n * (size_t)col] = dot3(v, ld3(cp + 15));
}

// ---- FP32 LU + FP64 iterative refinement ---------------------------------------
// The AIC (FP64, assembled once like the reference) is factored in FP32 with
// partial pivoting and inverted in FP32 (factor.cu); every solve then refines
// in FP64: x <- x + inv32 (b - A x), the residual b - A x in FP64.
// ||I - inv32 A|| ~ cond(A) x 2^-24 << 1 for vortex-lattice AICs, so each pass
// gains ~7 digits.
// Solve AIC gamVec = -RHS by refinement; records the final relative residual
// max|b - A x| / max|b| in s.luRes[0] and flags err[1] when it stays above 1e-9.
// One cluster of kSolveBlocks blocks, each with n / kSolveBlocks consecutive rows
// of the two products.  A thread takes a row and every S-th column of it, so that
// neighbouring threads read neighbouring rows of a column (the matrices are
// column-major); a warp then adds a row's S sums.  x and r go through global
// memory between the products and into every block's shared memory.  Bound by
// latency: six products of a few loads each and the cluster's barriers between
// them.  With a warp per row, each load of it 32 columns apart, 62 us at n = 300,
// now 42; on one SM it was 290.
constexpr int kRefinePasses = 3;
constexpr int kSolveBlocks = 8;
constexpr int kSolveThreads = 1024;
inline int solve_rows(int n) { return (n + kSolveBlocks - 1) / kSolveBlocks; }
inline int solve_slices(int n) { return std::max(1, std::min(n, kSolveThreads / solve_rows(n))); }
inline size_t solve_smem(int n) {
  return sizeof(double) * ((size_t)n + (size_t)solve_rows(n) * solve_slices(n)) + sizeof(float) * (size_t)n;
}
constexpr size_t kSolveSmemMax = sizeof(double) * (8192 + 1024) + sizeof(float) * 8192;  // at the most panels of a rotor
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__global__ void __cluster_dims__(kSolveBlocks, 1, 1) __launch_bounds__(kSolveThreads)
    k_solve_refine(Dims d, DevState s, int R, int S) {
  after_previous();
  const int n = d.n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * R, rows = max(0, min(R, n - row0));
  const double* rhs = s.RHS;
  volatile double* x = s.refX;
  volatile double* r = s.refR;
  extern __shared__ double vec[];   // the vector of the product at hand
  double* sums = vec + n;           // [slice][row]
  float* vec32 = reinterpret_cast<float*>(sums + R * S);
  __shared__ double red[32];
  // b = -RHS (under axisymmetry blade 1's for every blade), and its largest magnitude, in every block
  auto b = [&](int i) { return -1.0 * rhs[d.axisym ? i % d.npan : i]; };
  auto block_max = [&](double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = red[lane];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  };
  const int mr = threadIdx.x % R, ms = threadIdx.x / R;
  const bool mine = ms < S && mr < rows;
  double bmax = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = b(i);
    vec32[i] = (float)v;
    bmax = fmax(bmax, fabs(v));
  }
  bmax = block_max(bmax);
  for (int pass = 0; pass < kRefinePasses; ++pass) {
    if (pass) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) vec32[i] = (float)r[i];
      __syncthreads();
    }
    // x += inv32 r  (FP32 products of the FP32-rounded residual, FP64 update); r = b at first
    float* sums32 = reinterpret_cast<float*>(sums);
    if (mine) {
      const float* a = s.AICinv32 + row0 + mr;
      float z = 0.f;
#pragma unroll 8
      for (int j = ms; j < n; j += S) z = fmaf(a[(size_t)n * j], vec32[j], z);
      sums32[ms * R + mr] = z;
    }
    __syncthreads();
    for (int i = warp; i < rows; i += 32) {
      float z = 0.f;
      for (int k = lane; k < S; k += 32) z += sums32[k * R + i];
      for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      if (lane == 0) x[row0 + i] = (pass ? x[row0 + i] : 0.0) + (double)z;
    }
    cluster_sync();
    for (int i = threadIdx.x; i < n; i += blockDim.x) vec[i] = x[i];
    __syncthreads();
    // r = b - A x in FP64
    if (mine) {
      const double* a = s.AIC + row0 + mr;
      double ax = 0.0;
#pragma unroll 8
      for (int j = ms; j < n; j += S) ax = fma(a[(size_t)n * j], vec[j], ax);
      sums[ms * R + mr] = ax;
    }
    __syncthreads();
    for (int i = warp; i < rows; i += 32) {
      double ax = 0.0;
      for (int k = lane; k < S; k += 32) ax += sums[k * R + i];
      for (int o = 16; o > 0; o >>= 1) ax += __shfl_xor_sync(0xffffffffu, ax, o);
      if (lane == 0) r[row0 + i] = b(row0 + i) - ax;
    }
    cluster_sync();
  }
  if (blockIdx.x != 0) return;
  double rmax = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) rmax = fmax(rmax, fabs(r[i]));
  rmax = block_max(rmax);
  if (threadIdx.x == 0) {
    const double rel = bmax > 0.0 ? rmax / bmax : rmax;
    s.luRes[0] = rel;
    if (!(rel <= 1e-9)) atomicExch(s.err + 1, 12);
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    s.gamVecPrev[i] = s.gamVec[i];
    s.gamVec[i] = x[i];
  }
  // RHS keeps the reference's sign change (and, under axisymmetry, blade 1's rows in every blade)
  __syncthreads();
  if (d.axisym)
    for (int i = d.npan + threadIdx.x; i < n; i += blockDim.x) s.RHS[i] = s.RHS[i % d.npan];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) s.RHS[i] = -1.0 * s.RHS[i];
  for (int t = threadIdx.x; t < d.nb * d.npan; t += blockDim.x)
    if (t < d.nbC * d.npan || d.axisym) s.wGam[t] = x[d.axisym ? t % d.npan : t];
}

// ---- circulation solve (main.f90:522-603) ------------------------------------
__device__ __forceinline__ void rhs_row(const Dims& d, const DevState& s, const double* fr, int withWake, int t) {
  const double* w = panRec(d, fr, t / d.npan, t % d.npan);
  d3 v = ld3(w + 24);
  if (withWake) v = v + ld3(s.outv + 3 * (size_t)t);
  st3(s.velCP + 3 * (size_t)t, v);
  s.RHS[t] = dot3(v, ld3(w + 15));
}
__global__ void k_rhs(Dims d, DevState s, const double* fr, int withWake) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < d.nbC * d.npan) rhs_row(d, s, fr, withWake, t);
}
// A row a thread, its sum in order: bound by the rows' loads, 16 at a time (4 at a
// time, and with the RHS in a launch before, 11 us at 52 panels; a 40-step wing 9.66
// ms, now 9.59).  fr: the RHS of that frame first (null: it is there).
constexpr int kSolveRows = 1024;
__global__ void __launch_bounds__(kSolveRows) k_solve(Dims d, DevState s, const double* fr, int withWake) {
  after_previous();
  const int n = d.n;
  if (fr) {
    for (int t = threadIdx.x; t < d.nbC * d.npan; t += blockDim.x) rhs_row(d, s, fr, withWake, t);
    __syncthreads();
  }
  if (d.axisym)
    for (int r = d.npan + threadIdx.x; r < n; r += blockDim.x) s.RHS[r] = s.RHS[r % d.npan];
  __syncthreads();
  for (int r = threadIdx.x; r < n; r += blockDim.x) s.RHS[r] = -1.0 * s.RHS[r];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double sum = 0.0;
    const double* a = s.AICinv + i;
    int j = 0;
    constexpr int kB = 16;
    for (; j + kB <= n; j += kB) {
      double p[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) p[q] = a[(size_t)n * (j + q)] * s.RHS[j + q];
#pragma unroll
      for (int q = 0; q < kB; ++q) sum = sum + p[q];
    }
    for (; j < n; ++j) sum = sum + a[(size_t)n * j] * s.RHS[j];
    s.gamVecPrev[i] = s.gamVec[i];
    s.gamVec[i] = sum;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < d.nbC * d.npan; r += blockDim.x) s.wGam[r] = s.gamVec[r];
  __syncthreads();
  if (d.axisym)
    for (int r = d.npan + threadIdx.x; r < d.nb * d.npan; r += blockDim.x) s.wGam[r] = s.wGam[r % d.npan];
}

// ---- loads (main.f90:623-690, classdef.f90:1704-1896, 2196-2232, 4607-4671) ---
// Chunked (sum_chunk) accumulation of one component, as the oracle's ChunkSum
struct ChunkAcc1 {
  int C, cnt;
  double tot, part;
  __device__ ChunkAcc1(int c) : C(c), cnt(0), tot(0.0), part(0.0) {}
  // n values, 3 doubles apart
  __device__ void add(const exact64::Unit& u, const double* x, int n) {
    for (int i = 0; i < n;) {
      const int e = C > 0 ? min(n, i + C - cnt) : n;
      double p = C > 0 ? part : tot;
      cnt += e - i;
#pragma unroll 8
      for (; i < e; ++i) p = exact64::add(u, p, x[3 * i]);
      if (C <= 0) {
        tot = p;
      } else if (cnt == C) {
        tot = tot + p;
        part = 0.0;
        cnt = 0;
      } else {
        part = p;
      }
    }
  }
  __device__ double result() const { return (C > 0 && cnt > 0) ? tot + part : tot; }
};

// Sums over the rings of a rotor's blades at one collocation point, one block
// per point.  Every thread evaluates a ring (the four edges in vr_vind's order)
// and leaves its terms in shared memory -- the ring's (((f0 + f1) + f2) + f3) gam,
// its bound pair's (f1 + f3) gam and, on the trailing edge, f1 gam -- and lanes of
// eight warps add them in the reference's order, a lane per component and blade,
// so that only additions are serial.  A batch is up to kVcThreads rings: as many
// whole blades as fit (kVcBlades at most), or part of one.
//   bound: per blade s = 0, s + the pair's term panel by panel (spanwise
//          stations outer), s - the trailing-edge terms; blades added to 0
//          (rotor_vind_bywing_boundVortices, src/classdef.f90:1376-1393, 4445-4457)
//   wing:  per blade the rings' terms in summation blocks; blades added to 0
// Neighbouring rings of a blade share corners and edges where these hold bit for
// bit, as in a wake sheet: panel p's corner 3 and edge 3 are panel p - 1's corner
// 2 and edge 1, its corner 1 and edge 0 panel p - nc's corner 2 and edge 2, and
// an edge run backwards has the negated velocity.
// Bound by the FP64 unit at many points (300 points x 300 panels: 89 us with every
// ring on its own and the blades in turn, now 65), by one evaluation's chain and
// the longest blade's additions at few (16 points, two blades of 8: 37, now 28).
constexpr int kVcThreads = 256, kVcBlades = 32;
inline int velcp_blades(int npan) { return npan > kVcThreads ? 1 : std::min(kVcBlades, kVcThreads / npan); }
// of `te`: a group of blades has at most kVcThreads stations, one blade any number
inline size_t velcp_smem(int npan, int ns) {
  return sizeof(double) * 3 * (5 * (size_t)kVcThreads + 2 * kVcBlades + (size_t)velcp_blades(npan) * ns);
}
__device__ __forceinline__ bool same64(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ __forceinline__ bool same_point(const double* a, const double* b) {
  return same64(a[0], b[0]) && same64(a[1], b[1]) && same64(a[2], b[2]);
}
__device__ __forceinline__ d3 negated(const double* a) { return mk3(-a[0], -a[1], -a[2]); }
template <bool WING>
__device__ void ring_sums(const Dims& d, const DevState& s, const double* fr, d3 P, int sumChunk, int group, double* sm,
                          double& bound, double& wing) {
  constexpr int N = 3 * kVcThreads;
  double* ring = sm;             // [ring of the batch][component]
  double* pair = ring + N;
  double* U2 = pair + N;         // corner 2's unit vectors
  double* E1 = U2 + N;
  double* E2 = E1 + N;
  double* res = E2 + N;          // [bound, wing][blade of the group][component]
  double* te = res + 6 * kVcBlades;  // [blade of the group][station][component]
  const exact64::Unit u = exact64::load_unit();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npan = d.npan, nc = d.nc;
  bound = wing = 0.0;
  for (int b0 = 0; b0 < d.nb; b0 += group) {
    const int blades = min(group, d.nb - b0), total = blades * npan;
    double sb = 0.0;
    ChunkAcc1 acc(sumChunk);
    for (int q0 = 0; q0 < total; q0 += kVcThreads) {
      const int n = min(kVcThreads, total - q0), t = threadIdx.x;
      const bool live = t < n;
      const int k = live ? (q0 + t) / npan : 0, p = live ? (q0 + t) % npan : 0;
      const double* w = panRec(d, fr, b0 + k, p);
      const double* rv = s.wRvc + 4 * ((size_t)(b0 + k) * npan + p);
      corner64 c1, c2, c3;
      if (live) {
        c2 = exact64::make_corner(u, P, ld3(w + 6));
        st3(U2 + 3 * t, c2.u);
      }
      __syncthreads();
      bool s1 = false, s3 = false;  // corner 1 is panel p - nc's corner 2, corner 3 panel p - 1's
      d3 f1, f2;
      if (live) {
        const d3 p1 = ld3(w + 3), p3 = ld3(w + 9);
        s1 = p >= nc && t >= nc && same_point(w + 3, panRec(d, fr, b0 + k, p - nc) + 6);
        s3 = p % nc != 0 && t >= 1 && same_point(w + 9, panRec(d, fr, b0 + k, p - 1) + 6);
        if (s1) {
          c1.r = exact64::sub(u, P, p1);
          c1.u = ld3(U2 + 3 * (t - nc));
        } else {
          c1 = exact64::make_corner(u, P, p1);
        }
        f1 = exact64::vf_vind(u, c1, c2, rv[1]);
        st3(E1 + 3 * t, f1);
        if (s3) {
          c3.r = exact64::sub(u, P, p3);
          c3.u = ld3(U2 + 3 * (t - 1));
        } else {
          c3 = exact64::make_corner(u, P, p3);
        }
        if (WING) {
          f2 = exact64::vf_vind(u, c2, c3, rv[2]);
          st3(E2 + 3 * t, f2);
        }
      }
      __syncthreads();
      if (live) {
        const double g = s.wGam[(size_t)(b0 + k) * npan + p];
        const bool e0 = s1 && same_point(w, panRec(d, fr, b0 + k, p - nc) + 9) && same64(rv[0], rv[2 - 4 * nc]);
        const bool e3 = s3 && same_point(w, panRec(d, fr, b0 + k, p - 1) + 3) && same64(rv[3], rv[1 - 4]);
        corner64 c0;
        if (!e3 || (WING && !e0)) c0 = exact64::make_corner(u, P, ld3(w));
        const d3 f3 = e3 ? negated(E1 + 3 * (t - 1)) : exact64::vf_vind(u, c3, c0, rv[3]);
        if (WING) {
          const d3 f0 = e0 ? negated(E2 + 3 * (t - nc)) : exact64::vf_vind(u, c0, c1, rv[0]);
          st3(ring + 3 * t, exact64::mul(u, exact64::add(u, exact64::add(u, exact64::add(u, f0, f1), f2), f3), g));
        }
        st3(pair + 3 * t, exact64::mul(u, exact64::add(u, f1, f3), g));
        if (p % nc == nc - 1) st3(te + 3 * (k * d.ns + p / nc), exact64::mul(u, f1, g));
      }
      __syncthreads();
      // the blades' sums: bound by warps 0 to 3, wing by 4 to 7, every fourth blade each
      if (lane < 3 && (WING || warp < 4))
        for (int kb = warp & 3; kb < blades; kb += 4) {
          const int first = max(kb * npan, q0) - q0, last = min((kb + 1) * npan, q0 + n) - q0;
          if (first >= last) continue;
          const bool end = q0 + last == (kb + 1) * npan;
          if (warp >= 4) {
            acc.add(u, ring + 3 * first + lane, last - first);
            if (end) {
              res[3 * (kVcBlades + kb) + lane] = acc.result();
              acc = ChunkAcc1(sumChunk);
            }
          } else {
#pragma unroll 8
            for (int i = first; i < last; ++i) sb = exact64::add(u, sb, pair[3 * i + lane]);
            if (end) {
              const double* q = te + 3 * (size_t)kb * d.ns + lane;
#pragma unroll 8
              for (int j = 0; j < d.ns; ++j) sb = exact64::sub(u, sb, q[3 * j]);
              res[3 * kb + lane] = sb;
              sb = 0.0;
            }
          }
        }
      __syncthreads();
    }
    if (lane < 3)
      for (int kb = 0; kb < blades; ++kb) {
        bound = bound + res[3 * kb + lane];
        if (WING) wing = wing + res[3 * (kVcBlades + kb) + lane];
      }
    __syncthreads();
  }
}

// Velocity at the collocation points including the wing's own induced velocity
// minus its bound vortices (src/classdef.f90 calc_force's velCPTotal).
// fb (coupled rotors, else null): the bound-vortex velocity of every rotor
// at this rotor's collocation points, [rotor][point][xyz]; the entry of this
// rotor (self) is computed here.  velCPTotal = velCP - bound of every rotor in
// rotor order + this rotor's wing (src/main.f90:636-652).
__global__ void __launch_bounds__(kVcThreads) k_velcp_total(Dims d, DevState s, const double* fr, int sumChunk,
                                                            const double* fb, int nrs, int self, int group) {
  after_previous();
  extern __shared__ double sm[];
  const int t = blockIdx.x;
  const d3 P = ld3(panRec(d, fr, t / d.npan, t % d.npan) + 12);
  double bound, wing;
  ring_sums<true>(d, s, fr, P, sumChunk, group, sm, bound, wing);
  const int c = threadIdx.x;
  if (c < 3) {
    double v = s.velCP[3 * (size_t)t + c];
    if (fb) {
      const size_t M = (size_t)d.nbC * d.npan;
      for (int jr = 0; jr < nrs; ++jr) v = v - (jr == self ? bound : fb[3 * (jr * M + t) + c]);
    } else {
      v = v - bound;
    }
    v = v + wing;
    s.velCPTotal[3 * (size_t)t + c] = v;
  }
}

// Bound vortices of rotor (ds, ss, frs) at the collocation points of rotor
// (dt, frt), one block per point (a thread per point: 309 us at 16 panels).
__global__ void __launch_bounds__(kVcThreads) k_bound_foreign(Dims dt, const double* frt, Dims ds, DevState ss,
                                                              const double* frs, double* out, int group) {
  after_previous();
  extern __shared__ double sm[];
  const int t = blockIdx.x;
  const d3 P = ld3(panRec(dt, frt, t / dt.npan, t % dt.npan) + 12);
  double bound, wing;
  ring_sums<false>(ds, ss, frs, P, 0, group, sm, bound, wing);
  if (threadIdx.x < 3) out[3 * (size_t)t + threadIdx.x] = bound;
}

// ---- image rotors (src/classdef.f90:4990-5131) ------------------------------
// rotor_mirrorVelCP: the source's velCP with the image-plane component negated
__global__ void k_mirror_velcp(Dims d, DevState s, const double* src, int plane) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nb * d.npan) return;
  for (int c = 0; c < 3; ++c) {
    const double v = src[3 * (size_t)t + c];
    s.velCP[3 * (size_t)t + c] = c == plane - 1 ? -1.0 * v : v;
  }
}
// gamVecPrev = gamVec, rotor_mirrorGamma (gamVec = -source gamVec), map_gam
__global__ void k_mirror_gamma(Dims d, DevState s, const double* src) {
  after_previous();
  for (int i = threadIdx.x; i < d.n; i += blockDim.x) {
    s.gamVecPrev[i] = s.gamVec[i];
    s.gamVec[i] = -1.0 * src[i];
  }
  __syncthreads();
  for (int r = threadIdx.x; r < d.nbC * d.npan; r += blockDim.x) s.wGam[r] = s.gamVec[r];
  __syncthreads();
  if (d.axisym)
    for (int r = d.npan + threadIdx.x; r < d.nb * d.npan; r += blockDim.x) s.wGam[r] = s.wGam[r % d.npan];
}
// rotor_mirrorWake: mode 0 the active current wake, 1 the active predicted
// wake (node positions; the predicted wake's circulation and cores are the
// current ones, which already mirror the source's), 2 every row of the
// current wake; node coordinates in the image plane and circulation negated
// (vr_mirror, Fwake_mirror: src/classdef.f90:722-735, 982-993)
__global__ void k_mirror_wake(Dims d, DevState dst, DevState src, int mode, int rowNear, int rowFar, int plane) {
  after_previous();
  const int r0 = mode == 2 ? 0 : rowNear - 1, f0 = mode == 2 ? 0 : rowFar - 1;
  const long nNear = (long)d.nb * (d.NW - r0) * d.ns;
  const long nFar = d.NF - f0 > 0 ? (long)d.nb * (d.NF - f0) : 0;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int k0 = plane - 1;
  if (t < nNear) {
    const int rows = d.NW - r0;
    const int b = (int)(t / ((long)rows * d.ns)), rem = (int)(t % ((long)rows * d.ns));
    const int j = rem / rows, i = r0 + rem % rows;
    const size_t idx = ringI(d, b, i, j);
    const double* sc = (mode == 1 ? src.nCP : src.nC) + 12 * idx;
    double* dc = (mode == 1 ? dst.nCP : dst.nC) + 12 * idx;
    for (int k = 0; k < 12; ++k) dc[k] = k % 3 == k0 ? -1.0 * sc[k] : sc[k];
    if (mode != 1) {
      dst.nGam[idx] = -1.0 * src.nGam[idx];
      for (int q = 0; q < 4; ++q) dst.nRvc[4 * idx + q] = src.nRvc[4 * idx + q];
      dst.nAge[idx] = src.nAge[idx];
    }
  } else if (t < nNear + nFar) {
    const long u = t - nNear;
    const int b = (int)(u / (d.NF - f0)), i = f0 + (int)(u % (d.NF - f0));
    const size_t f = (size_t)b * d.NF + i;
    const double* sc = (mode == 1 ? src.fCP : src.fC) + 6 * f;
    double* dc = (mode == 1 ? dst.fCP : dst.fC) + 6 * f;
    for (int k = 0; k < 6; ++k) dc[k] = k % 3 == k0 ? -1.0 * sc[k] : sc[k];
    if (mode != 1) {
      dst.fGam[f] = -1.0 * src.fGam[f];
      dst.fRvc[f] = src.fRvc[f];
      dst.fRvc0[f] = src.fRvc0[f];
      dst.fL0[f] = src.fL0[f];
      dst.fLc[f] = src.fLc[f];
      dst.fAge[f] = src.fAge[f];
    }
  }
}

// velCP = kinematic velocity + each term in turn (coupled rotors:
// src/main.f90:549-561, the wake of every rotor and the wing of the others,
// one per-rotor sum per term); RHS = velCP . nCap
__global__ void k_rhs_terms(Dims d, DevState s, const double* fr, const double* terms, int nterms, int M) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nbC * d.npan) return;
  const double* w = panRec(d, fr, t / d.npan, t % d.npan);
  d3 v = ld3(w + 24);
  for (int k = 0; k < nterms; ++k) v = v + ld3(terms + 3 * ((size_t)k * M + t));
  st3(s.velCP + 3 * (size_t)t, v);
  s.RHS[t] = dot3(v, ld3(w + 15));
}

// libMath.f90:293-426 (Doolittle inverse of lsq2's 3x3 normal matrix; its
// pivot search never swaps rows for these matrices)
__device__ void inv3_doolittle(const double* A, double* X) {
  double L[9], U[9];
  for (int k = 0; k < 9; ++k) L[k] = U[k] = 0.0;
  auto at = [](int i, int j) { return i + 3 * j; };
  for (int j = 0; j < 3; ++j) U[at(0, j)] = A[at(0, j)];
  for (int i = 0; i < 3; ++i) L[at(i, 0)] = A[at(i, 0)] / A[at(0, 0)];
  for (int i = 1; i < 3; ++i)
    for (int j = 1; j < 3; ++j) {
      double su = 0.0, sl = 0.0;
      for (int k = 0; k < i; ++k) {
        su = su + L[at(i, k)] * U[at(k, j)];
        sl = sl + L[at(j, k)] * U[at(k, i)];
      }
      U[at(i, j)] = A[at(i, j)] - su;
      if (fabs(U[at(i, i)]) > kEps) L[at(j, i)] = (A[at(j, i)] - sl) / U[at(i, i)];
    }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      if (i > j) U[at(i, j)] = 0.0;
      else if (j > i) L[at(i, j)] = 0.0;
    }
  for (int bb = 0; bb < 3; ++bb) {
    double Pb[3], dd[3], x[3];
    for (int i = 0; i < 3; ++i) {
      double sum = 0.0;
      for (int k = 0; k < 3; ++k) sum = sum + (i == k ? 1.0 : 0.0) * (k == bb ? 1.0 : 0.0);
      Pb[i] = sum;
    }
    dd[0] = Pb[0];
    for (int i = 1; i < 3; ++i) {
      double sum = 0.0;
      for (int k = 0; k < i; ++k) sum = sum + L[at(i, k)] * dd[k];
      dd[i] = Pb[i] - sum;
    }
    x[2] = dd[2] / U[at(2, 2)];
    for (int i = 1; i >= 0; --i) {
      double sum = 0.0;
      for (int k = i + 1; k < 3; ++k) sum = sum + U[at(i, k)] * x[k];
      x[i] = (dd[i] - sum) / U[at(i, i)];
    }
    for (int i = 0; i < 3; ++i) X[at(i, bb)] = x[i];
  }
}

// libMath.f90:577-605, for the three components of one section: the normal
// matrix and its inverse are the stations' alone
struct Lsq2 {
  double s1 = 0, s2 = 0, Ai[9];
  __device__ void stations(const double* xd, int n) {
    double s3 = 0, s4 = 0;
    for (int i = 0; i < n; ++i) {
      const double x = xd[i];
      s1 = s1 + x;
      s2 = s2 + x * x;
      s3 = s3 + (x * x) * x;
      s4 = s4 + pow4(x);
    }
    const double A[9] = {(double)n, s1, s2, s1, s2, s3, s2, s3, s4};
    inv3_doolittle(A, Ai);
  }
  __device__ double at(double xq, const double* xd, const double* yd, int ystride, int n) const {
    double r1 = 0, r2 = 0, r3 = 0;
    for (int i = 0; i < n; ++i) {
      const double x = xd[i], y = yd[i * ystride];
      r1 = r1 + y;
      r2 = r2 + y * x;
      r3 = r3 + y * (x * x);
    }
    double c[3];
    for (int i = 0; i < 3; ++i) c[i] = Ai[i] * r1 + Ai[i + 3] * r2 + Ai[i + 6] * r3;
    return c[0] + c[1] * xq + (c[2] * xq) * xq;
  }
};

constexpr int kMaxNc = 64;

__global__ void k_step_begin(Dims d, DevState s) {
  after_previous();
  const int it = s.devIter[0] + 1;
  const double* src = s.frames + (size_t)it * d.fl.size;
  for (int i = threadIdx.x; i < d.fl.size; i += blockDim.x) s.curFrame[i] = src[i];
  __syncthreads();
  if (threadIdx.x == 0) s.devIter[0] = it;
}

// ---- airfoil tables (libC81.f90:190-351) ------------------------------------
// interval of x in the ascending axis A[0..n): 1-based (i1, i2) as the
// reference's binary search leaves them, ends snapped within the
// single-precision epsilon
__device__ void c81_interval(const double* A, int n, double x, int& i1, int& i2) {
  i1 = 1;
  i2 = n;
  while (i1 != i2 && i2 != i1 + 1) {
    const int i = (i1 + i2) / 2;
    if (x < A[i - 1]) i2 = i;
    else if (x > A[i - 1]) i1 = i;
    else i1 = i2 = i;
  }
  const double epsf = 1.1920928955078125e-07;  // epsilon(1.) of the default real kind
  if (fabs(A[i1 - 1] - x) <= epsf) i2 = i1;
  else if (fabs(A[i2 - 1] - x) <= epsf) i1 = i2;
}
// coefficient c (0 lift, 1 drag, 2 moment) of table T at (alpha degrees, Mach)
__device__ double c81_get(const double* T, int c, double alpha, double mach) {
  size_t o = 6;
  int nm = 0, na = 0;
  for (int k = 0; k <= c; ++k) {
    nm = (int)T[2 * k];
    na = (int)T[2 * k + 1];
    if (k < c) o += (size_t)nm + na + (size_t)nm * na;
  }
  const double* Ma = T + o;
  const double* A = Ma + nm;
  const double* C = A + na;
  int a1, a2, m1, m2;
  c81_interval(A, na, alpha, a1, a2);
  c81_interval(Ma, nm, mach, m1, m2);
  auto v = [&](int i, int j) { return C[(i - 1) + (size_t)na * (j - 1)]; };
  if (a1 == a2) {
    if (m1 == m2) return v(a1, m1);
    return v(a1, m1) + ((mach - Ma[m1 - 1]) * (v(a1, m2) - v(a1, m1))) / (Ma[m2 - 1] - Ma[m1 - 1]);
  }
  if (m1 == m2) return v(a1, m1) + ((alpha - A[a1 - 1]) * (v(a2, m1) - v(a1, m1))) / (A[a2 - 1] - A[a1 - 1]);
  const double y2m = Ma[m2 - 1] - mach, my1 = mach - Ma[m1 - 1];
  const double lo = v(a1, m1) * y2m + v(a1, m2) * my1;
  const double hi = v(a2, m1) * y2m + v(a2, m2) * my1;
  const double num = (A[a2 - 1] - alpha) * lo + (alpha - A[a1 - 1]) * hi;
  return num / (A[a2 - 1] - A[a1 - 1]) / (Ma[m2 - 1] - Ma[m1 - 1]);
}

// One block.  FP64 work is 64 cycles an instruction and its divisions and roots
// hundreds, so each phase runs over the smallest independent items -- panels,
// (section, component), sections, (blade, component) -- with the integer
// divisions; only the ordered sums are serial.  (Over sections alone, with
// CUDA's divisions, it took 90 us at 75 sections of 4 blades and 84 us at 13
// sections of 4 panels.)  tmp: 9 doubles a panel.
constexpr int kLoadsThreads = 512;
__global__ void __launch_bounds__(kLoadsThreads) k_loads(Dims d, DevState s, const double* fr, int iter) {
  after_previous();
  if (iter < 0) iter = s.devIter[0];
  const int nsec = d.nbC * d.ns, npan = d.nbC * d.npan;
  const double iGS = -1.0 * fsign1(d.omega);
  double* tmp = s.loadTmp;
  // phase A: sectional resultant velocity and lift/drag directions
  for (int gp = threadIdx.x; gp < npan; gp += blockDim.x) {
    const int b = gp / d.npan, p = gp % d.npan;
    const double* w = panRec(d, fr, b, p);
    st3(tmp + 9 * (size_t)gp, exact64::noproj(ld3(s.velCPTotal + 3 * (size_t)gp), ld3(w + 21)));
    const double* sec = fr + d.fl.sec + ((size_t)b * d.ns + p / d.nc) * kSec;
    tmp[9 * (size_t)gp + 3] = dot3(ld3(w + 12) - ld3(sec + 9), ld3(sec));
  }
  __syncthreads();
  for (int t3 = threadIdx.x; t3 < 3 * nsec; t3 += blockDim.x) {
    const int t = t3 / 3, c = t3 % 3, b = t / d.ns, is = t % d.ns;
    const double* q = tmp + 9 * ((size_t)b * d.npan + (size_t)d.nc * is);
    double v;
    if (d.nc >= 3) {
      const double* sec = fr + d.fl.sec + ((size_t)b * d.ns + is) * kSec;
      double xd[kMaxNc];
      for (int ic = 0; ic < d.nc; ++ic) xd[ic] = q[9 * ic + 3];
      const double xq = dot3(ld3(sec + 6) - ld3(sec + 9), ld3(sec));
      Lsq2 fit;
      fit.stations(xd, d.nc);
      v = fit.at(xq, xd, q + c, 9, d.nc);
    } else {
      double sum = 0.0;
      for (int ic = 0; ic < d.nc; ++ic) sum = sum + q[9 * ic + c];
      v = sum / (double)d.nc;
    }
    s.secResVel[t3] = v;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nsec; t += blockDim.x) {
    const d3 dd = exact64::unit(ld3(s.secResVel + 3 * (size_t)t));
    const d3 yAF = ld3(fr + d.fl.ax + 9 * (t / d.ns) + 3);
    st3(s.secDragDir + 3 * (size_t)t, dd);
    st3(s.secLiftDir + 3 * (size_t)t, fsign1(d.omega) * exact64::unit(cross3(dd, yAF)));
  }
  __syncthreads();
  // phase B with airfoil tables (forceCalcSwitch 1: blade_calc_force_alpha,
  // src/classdef.f90:2091-2105, 2146-2195, 2234-2250): sectional angle of
  // attack from the resultant velocity, CL and CD from the section's table
  // at that angle and Mach number, lift along the lift direction, the
  // inertial force along y x V with the sign of the section's circulation;
  // the sectional drag stays zero (the reference never assigns it here) and
  // the panel pressures and gamPrev are not computed.
  for (int t = threadIdx.x; d.forceCalc == 1 && t < nsec; t += blockDim.x) {
    const int b = t / d.ns, is = t % d.ns;
    const double* sec = fr + d.fl.sec + ((size_t)b * d.ns + is) * kSec;
    const d3 rv = ld3(s.secResVel + 3 * (size_t)t);
    const double alpha = atan2(dot3(rv, ld3(sec + 3)), dot3(rv, ld3(sec)));
    const double m = norm3(rv);
    const double* T = s.c81 + s.c81Off[s.airfoilNo[t]];
    const double aDeg = alpha * kRad2Deg, mach = m / d.velSound;
    const double cl = c81_get(T, 0, aDeg, mach);
    const double cd = c81_get(T, 1, aDeg, mach);
    const double lead = ((0.5 * d.density) * (m * m)) * s.secArea[t];
    const d3 liftDir = ld3(s.secLiftDir + 3 * (size_t)t);
    const d3 sL = (liftDir * lead) * cl;
    const d3 sLU = (liftDir * lead) * 0.0;
    double gs = 0.0;
    for (int ic = 0; ic < d.nc; ++ic) gs = gs + s.wGam[(size_t)b * d.npan + ic + d.nc * is];
    const d3 yAF = ld3(fr + d.fl.ax + 9 * b + 3);
    d3 fi = fsign1(gs) * unit3(cross3(yAF, rv));
    fi = norm3(sL) * fi;
    fi = fi + 0.0 * unit3(rv);
    st3(s.secForceInertial + 3 * (size_t)t, fi);
    st3(s.secLift + 3 * (size_t)t, sL);
    st3(s.secLiftUnsteady + 3 * (size_t)t, sLU);
    s.secCL[t] = cl;
    s.secCD[t] = cd;
    s.secCLu[t] = 0.0;
  }
  // phase B: panel pressures and sectional forces (blade_calc_force)
  if (d.forceCalc != 1) {
    for (int gp = threadIdx.x; gp < npan; gp += blockDim.x) {
      const int b = gp / d.npan, p = gp % d.npan, is = p / d.nc, ic = p % d.nc;
      const d3 liftDir = ld3(s.secLiftDir + 3 * ((size_t)b * d.ns + is));
      const double* w = panRec(d, fr, b, p);
      const d3 velCP = ld3(s.velCP + 3 * (size_t)gp);
      const double vTC = dot3(velCP, ld3(w + 18));
      const double vTS = dot3(velCP, ld3(w + 21));
      const double g = s.wGam[gp];
      double gEC = ic == 0 ? g : g - s.wGam[gp - 1];
      double gES = is == 0 ? g : g - s.wGam[gp - d.nc];
      gEC = iGS * gEC;
      gES = iGS * gES;
      const double gamTrapz = ic > 0 ? (iGS * 0.5) * (g + s.wGam[gp - 1]) : (iGS * 0.5) * g;
      const double delPU = exact64::quotient(d.density * (gamTrapz - s.gamPrev[gp]), d.dt);
      double delP = delPU + exact64::quotient(d.density * vTC * gEC, s.panMeanChord[gp]);
      if (d.spanwiseLift != 0) delP = delP + exact64::quotient(d.density * vTS * gES, s.panMeanSpan[gp]);
      s.gamPrev[gp] = gamTrapz;
      const d3 nCap = ld3(w + 15);
      const d3 nF = (delP * s.panArea[gp]) * nCap;
      const d3 nFU = (delPU * s.panArea[gp]) * nCap;
      st3(tmp + 9 * (size_t)gp, nF);
      st3(tmp + 9 * (size_t)gp + 3, exact64::proj(nF, liftDir));
      st3(tmp + 9 * (size_t)gp + 6, exact64::proj(nFU, liftDir));
    }
    __syncthreads();
    for (int t9 = threadIdx.x; t9 < 9 * nsec; t9 += blockDim.x) {
      const int t = t9 / 9, c = t9 % 9;
      const double* q = tmp + 9 * ((size_t)(t / d.ns) * d.npan + (size_t)d.nc * (t % d.ns)) + c;
      double sum = 0.0;
      for (int ic = 0; ic < d.nc; ++ic) sum = sum + q[9 * ic];
      double* o = c < 3 ? s.secForceInertial : c < 6 ? s.secLift : s.secLiftUnsteady;
      o[3 * (size_t)t + c % 3] = sum;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nsec; t += blockDim.x) {
      const int b = t / d.ns;
      const d3 xAF = ld3(fr + d.fl.ax + 9 * b), zAF = ld3(fr + d.fl.ax + 9 * b + 6);
      const d3 sL = ld3(s.secLift + 3 * (size_t)t), sLU = ld3(s.secLiftUnsteady + 3 * (size_t)t);
      st3(s.secLiftInPlane + 3 * (size_t)t, iGS * exact64::proj(sL, xAF));
      st3(s.secLiftOutPlane + 3 * (size_t)t, exact64::proj(sL, zAF));
      const double m = exact64::norm(ld3(s.secResVel + 3 * (size_t)t));
      const double q = (0.5 * d.density) * (m * m);
      const double area = s.secArea[t];
      if (fabs(q) > kEps) {
        const double sg = fsign1(dot3(sL, zAF));
        s.secCL[t] = exact64::quotient(exact64::norm(sL) * sg, q * area);
        s.secCD[t] = 0.0 / (q * area);
        s.secCLu[t] = exact64::quotient(exact64::norm(sLU) * sg, q * area);
      } else {
        s.secCL[t] = s.secCD[t] = s.secCLu[t] = 0.0;
      }
    }
  }
  __syncthreads();
  // phase C: blade sums (blade_sumSecToNetForces), one component a thread
  for (int t9 = threadIdx.x; t9 < 9 * d.nbC; t9 += blockDim.x) {
    const int b = t9 / 9, c = t9 % 9;
    const double* q = (c < 3 ? s.secForceInertial : c < 6 ? s.secLift : s.secLiftUnsteady) + 3 * (size_t)b * d.ns + c % 3;
    double sum = 0.0;
#pragma unroll 8
    for (int is = 0; is < d.ns; ++is) sum = sum + q[3 * is];
    s.bladeForce[12 * (size_t)b + (c < 6 ? c : c + 3)] = sum;
    if (c < 3) s.bladeForce[12 * (size_t)b + 6 + c] = 0.0;
  }
  __syncthreads();
  // phase D: rotor sums and the CT row (rotor_sumBladeToNetForces, force2file)
  __shared__ double net[9];  // inertial, lift, unsteady lift
  if (threadIdx.x < 9) {
    const int c = threadIdx.x, o = c < 6 ? c : c + 3;
    double sum = 0.0;
    if (d.axisym) {
      sum = (double)d.nb * s.bladeForce[o];
    } else {
      for (int b = 0; b < d.nbC; ++b) sum = sum + s.bladeForce[12 * (size_t)b + o];
    }
    net[c] = sum;
    if (c < 6) s.rotorLift[c < 3 ? c + 3 : c - 3] = sum;
  }
  __syncthreads();
  if (threadIdx.x < 10) {
    const double D = d.nonDimDenom;
    double v = 0.0;
    if (threadIdx.x == 1) v = fsign1(dot3(ld3(net + 3), ld3(fr + d.fl.rot))) * exact64::norm(ld3(net + 3));
    if (threadIdx.x == 3) v = exact64::norm(ld3(net + 6));
    if (threadIdx.x >= 7) v = net[threadIdx.x - 7];
    s.ctHist[10 * (size_t)iter + threadIdx.x] = threadIdx.x == 0 ? (double)iter : v / D;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
void launch_shed(const Dims& d, const DevState& s, const double* frame, int rowNear, cudaStream_t st) {
  count_launch();
  launch_next(k_shed, nblk(d.nb * d.ns, 128), 128, 0, st, d, s, frame, rowNear);
}
static long wake_items(const Dims& d, int rowNear, int rowFar) {
  return (long)d.nb * (d.NW - (rowNear - 1)) * d.ns + (long)d.nb * std::max(d.NF - (rowFar - 1), 0);
}
void launch_wake_begin(const Dims& d, const DevState& s, const double* frame, int rowNear, int rowFar, bool dissipate,
                       cudaStream_t st) {
  const long n = wake_items(d, rowNear, rowFar);
  if (n <= 0) return;
  count_launch();
  launch_next(k_wake_begin, nblk(n, 128), 128, 0, st, d, s, frame, rowNear, rowFar, dissipate ? 1 : 0);
}
void launch_predict(const Dims& d, const DevState& s, int rowNear, int rowFar, cudaStream_t st) {
  const long n = wake_items(d, rowNear, rowFar) + (rowNear > 1 ? (long)d.nb * d.ns : 0);
  if (n <= 0) return;
  count_launch();
  launch_next(k_predict, nblk(n, 128), 128, 0, st, d, s, rowNear, rowFar);
}
void launch_correct(const Dims& d, const DevState& s, const double* frame, int rowNear, int rowFar, bool strain, int op,
                    cudaStream_t st) {
  const long n = wake_items(d, rowNear, rowFar);
  if (n > 0) {
    count_launch();
    launch_next(k_correct, nblk(n, 128), 128, 0, st, d, s, rowNear, rowFar, strain ? 1 : 0);
  }
  const int rollBlocks = rowNear == 1 && d.NF > 0 ? nblk(d.nb, 4) : 0;
  const long m = n + (rowNear > 1 ? (long)d.nb * d.ns : 0) +
                 (op >= 0 ? (long)d.nb * d.NW * (d.ns + 1) * 3 + (long)d.nb * d.NF * 3 : 0);
  if (m + rollBlocks <= 0) return;
  count_launch();
  launch_next(k_correct_back, rollBlocks + nblk(m, 128), 128, 0, st, d, s, frame, rowNear, rowFar, op, rollBlocks);
}
void launch_copy_predicted(const Dims& d, const DevState& s, int rowNear, int rowFar, cudaStream_t st) {
  const long n = (long)d.nbC * (d.NW - (rowNear - 1)) * d.ns + (long)d.nbC * (d.NF - (rowFar - 1) > 0 ? d.NF - (rowFar - 1) : 0);
  if (n > 0) {
    count_launch();
    launch_next(k_copy_pred, nblk(n, 256), 256, 0, st, d, s, rowNear, rowFar);
  }
}
void launch_convect(const Dims& d, const DevState& s, const double* frame, int rowNear, int rowFar, bool pred,
                    cudaStream_t st) {
  const int rowsF = d.NF - (rowFar - 1) > 0 ? d.NF - (rowFar - 1) : 0;
  const long n1 = (long)d.nbC * (pred ? 1 : d.NW - (rowNear - 1)) * (d.ns + 1) + (long)d.nbC * rowsF;
  if (n1 > 0) {
    count_launch();
    launch_next(k_shift, nblk(n1, 256), 256, 0, st, d, s, rowNear, rowFar, pred ? 1 : 0);
  }
  const long n2 = (long)d.nbC * (d.NW - (rowNear - 1)) * d.ns + (long)d.nbC * (d.NF - rowFar > 0 ? d.NF - rowFar : 0);
  if (n2 > 0) {
    count_launch();
    launch_next(k_continuity, nblk(n2, 256), 256, 0, st, d, s, rowNear, rowFar, pred ? 1 : 0);
  }
  if (d.axisym && d.nb > 1) {
    const long n3 = (long)(d.nb - 1) * (d.NW - (rowNear - 1)) * d.ns + (long)(d.nb - 1) * rowsF;
    if (n3 > 0) {
      count_launch();
      launch_next(k_axisym, nblk(n3, 256), 256, 0, st, d, s, frame, rowNear, rowFar, pred ? 1 : 0);
    }
  }
}
void launch_presc_update(const Dims& d, const DevState& s, const double* frame, int rowFar, bool pred,
                         cudaStream_t st) {
  if (!s.pfC || d.NF - (rowFar - 1) < 1) return;
  count_launch();
  launch_next(k_presc_update, d.nbC, 256, 0, st, d, s, frame, rowFar, pred ? 1 : 0);
  if (d.axisym && d.nb > 1) {
    count_launch();
    launch_next(k_presc_axisym, nblk((long)(d.nb - 1) * kPresc, 256), 256, 0, st, d, s, frame, pred ? 1 : 0);
  }
}
void launch_burst(const Dims& d, const DevState& s, int rowFar, cudaStream_t st) {
  const long n = (long)d.nb * (d.NF - (rowFar - 1) - 1);
  if (n > 0) {
    count_launch();
    launch_next(k_burst, nblk(n, 256), 256, 0, st, d, s, rowFar);
  }
}
void launch_strain(const Dims& d, const DevState& s, int rowFar, cudaStream_t st) {
  const long n = (long)d.nb * (d.NF - (rowFar - 1));
  if (n > 0) {
    count_launch();
    launch_next(k_strain, nblk(n, 256), 256, 0, st, d, s, rowFar);
  }
}
void launch_rollup(const Dims& d, const DevState& s, int rowFar, cudaStream_t st) {
  int rowFarNext = rowFar - 1;
  if (d.NF > 0 && rowFarNext == 0) {
    const long n = (long)d.nb * d.NF;
    count_launch();
    launch_next(k_far_to_tmp, nblk(n, 256), 256, 0, st, d, s);
    count_launch();
    launch_next(k_far_from_tmp, nblk(n, 256), 256, 0, st, d, s);
    rowFarNext = 1;
  }
  count_launch();
  launch_next(k_rollup, nblk(d.nb, 32), 32, 0, st, d, s, rowFarNext);
  const long n = (long)d.nb * d.NW * d.ns;
  count_launch();
  launch_next(k_near_to_tmp, nblk(n, 256), 256, 0, st, d, s);
  count_launch();
  launch_next(k_near_from_tmp, nblk(n, 256), 256, 0, st, d, s);
}
void launch_velop(const Dims& d, const DevState& s, VelOp op, cudaStream_t st) {
  const long nN = (long)d.nbC * d.NW * (d.ns + 1) * 3, nF = (long)d.nbC * d.NF * 3;
  if (nN + nF > 0) {
    count_launch();
    launch_next(k_velop, nblk(nN + nF, 256), 256, 0, st, s, nN, nF, (int)op);
  }
}
void launch_order2(const Dims& d, const DevState& s, int rowNear, int rowFar, cudaStream_t st) {
  const long n = (long)d.nbC * (d.ns + 1) * (d.NW - (rowNear - 1)) * 3 +
                 (long)d.nbC * (d.NF - (rowFar - 1) > 0 ? d.NF - (rowFar - 1) : 0) * 3;
  if (n <= 0) return;
  count_launch();
  launch_next(k_order2, nblk(n, 256), 256, 0, st, d, s, rowNear, rowFar, 0);
  count_launch();
  launch_next(k_order2, nblk(n, 256), 256, 0, st, d, s, rowNear, rowFar, 1);
}
int node_target_count(const Dims& d, int rowNear, int rowFar) {
  const int rowsN = d.NW - (rowNear - 1);
  const int rowsF = d.NF - (rowFar - 1) > 0 ? d.NF - (rowFar - 1) : 0;
  return d.nbC * (rowsN * (d.ns + 1) + rowsF);
}
void launch_scatter_nodes(const Dims& d, const DevState& s, const double* frame, int rowNear, int rowFar, bool pred,
                          double initWakeVel, int op, cudaStream_t st) {
  const int M = node_target_count(d, rowNear, rowFar);
  const int addInit = initWakeVel != 0.0 ? 1 : 0;
  if (M > 0) {
    count_launch();
    launch_next(k_scatter_nodes, nblk(M, 256), 256, 0, st, d, s, frame, rowNear, rowFar, pred ? 1 : 0, initWakeVel,
                addInit, op, M);
  }
}
void launch_aic(const Dims& d, const DevState& s, const double* frame, cudaStream_t st) {
  const long n = (long)d.n * d.n;
  count_launch();
  launch_next(k_aic, nblk(n, 128), 128, 0, st, d, s, frame);
}
static void solve_refine(const Dims& d, const DevState& s, cudaStream_t st) {
  const size_t smem = solve_smem(d.n);
  if (smem > 40 * 1024)
    cudaFuncSetAttribute(k_solve_refine, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSolveSmemMax);
  launch_next(k_solve_refine, kSolveBlocks, kSolveThreads, smem, st, d, s, solve_rows(d.n), solve_slices(d.n));
}
void launch_solve(const Dims& d, const DevState& s, const double* frame, bool withWake, cudaStream_t st) {
  const int rows = d.nbC * d.npan;
  count_launch();
  if (!s.LU32 && rows <= kSolveRows) {
    launch_next(k_solve, 1, kSolveRows, 0, st, d, s, frame, withWake ? 1 : 0);
    return;
  }
  launch_next(k_rhs, nblk(rows, 128), 128, 0, st, d, s, frame, withWake ? 1 : 0);
  count_launch();
  if (s.LU32) solve_refine(d, s, st);
  else launch_next(k_solve, 1, kSolveRows, 0, st, d, s, nullptr, 0);
}
void launch_step_begin(const Dims& d, const DevState& s, cudaStream_t st) {
  count_launch();
  launch_next(k_step_begin, 1, 1024, 0, st, d, s);
}
void launch_rhs_terms(const Dims& d, const DevState& s, const double* frame, const double* terms, int nterms,
                      cudaStream_t st) {
  count_launch();
  launch_next(k_rhs_terms, nblk(d.nbC * d.npan, 128), 128, 0, st, d, s, frame, terms, nterms, d.nbC * d.npan);
}
void launch_mirror_velcp(const Dims& d, const DevState& s, const double* srcVelCP, int plane, cudaStream_t st) {
  count_launch();
  launch_next(k_mirror_velcp, nblk(d.nb * d.npan, 128), 128, 0, st, d, s, srcVelCP, plane);
}
void launch_mirror_gamma(const Dims& d, const DevState& s, const double* srcGamVec, cudaStream_t st) {
  count_launch();
  launch_next(k_mirror_gamma, 1, 1024, 0, st, d, s, srcGamVec);
}
void launch_mirror_wake(const Dims& d, const DevState& dst, const DevState& src, int mode, int rowNear, int rowFar,
                        int plane, cudaStream_t st) {
  const int r0 = mode == 2 ? 0 : rowNear - 1, f0 = mode == 2 ? 0 : rowFar - 1;
  const long n = (long)d.nb * (d.NW - r0) * d.ns + (d.NF - f0 > 0 ? (long)d.nb * (d.NF - f0) : 0);
  if (n <= 0) return;
  count_launch();
  launch_next(k_mirror_wake, nblk(n, 256), 256, 0, st, d, dst, src, mode, rowNear, rowFar, plane);
}
void launch_solve_only(const Dims& d, const DevState& s, cudaStream_t st) {
  count_launch();
  if (s.LU32) solve_refine(d, s, st);
  else launch_next(k_solve, 1, kSolveRows, 0, st, d, s, nullptr, 0);
}
// shared memory for up to 8192 stations (the most panels a rotor has)
static void velcp_attr() {
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && attr[dev].load(std::memory_order_acquire)) return;
  const int most = (int)velcp_smem(8192, 8192);
  cudaFuncSetAttribute(k_velcp_total, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  cudaFuncSetAttribute(k_bound_foreign, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
}
void launch_bound_foreign(const Dims& dt, const double* frameT, const Dims& ds, const DevState& ss,
                          const double* frameS, double* out, cudaStream_t st) {
  count_launch();
  velcp_attr();
  launch_next(k_bound_foreign, dt.nbC * dt.npan, kVcThreads, velcp_smem(ds.npan, ds.ns), st, dt, frameT, ds, ss, frameS, out,
              velcp_blades(ds.npan));
}
void launch_loads(const Dims& d, const DevState& s, const double* frame, int sumChunk, int iter, cudaStream_t st,
                  const double* foreignBound, int nrs, int self) {
  count_launch();
  velcp_attr();
  launch_next(k_velcp_total, d.nbC * d.npan, kVcThreads, velcp_smem(d.npan, d.ns), st, d, s, frame, sumChunk, foreignBound,
              nrs, self, velcp_blades(d.npan));
  count_launch();
  launch_next(k_loads, 1, kLoadsThreads, 0, st, d, s, frame, iter);
}

}  // namespace vlm
