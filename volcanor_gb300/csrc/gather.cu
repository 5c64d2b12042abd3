// Source records and targets of a solver evaluation, gathered from a case's
// state in one launch: FP64 records, in the FP32 precisions their lattice edge
// weights and FP32 records, the wake-node or collocation-point targets, and the
// near-pair counters reset.  Four lanes a record, one corner and edge each.
// (A thread per record walked 18 doubles and four FP64-compared neighbours, a
// second kernel packed the records, a third wrote the targets and a fill reset
// the counter: 8 + 12.5 + 1.6 + 1.2 us at 500 records and the launches between.)
// In FP64 it also marks what neighbouring rings of a sheet share (a launch of its own
// before each evaluation took 4.6 us).
// Only copies and one FP64 subtraction are rounded here, so the unit shares the FP32
// kernels' compiler options.
#include "launch.h"
#include "pack32.h"
#include "state_dev.h"
#include "vlm_bs.h"
#include "vlm_math.h"
#include "vlm_solver.h"

namespace vlm {

namespace {

// a == b for numbers, on the integer units
__device__ __forceinline__ bool same(double a, double b) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(a), y = (unsigned long long)__double_as_longlong(b);
  return x == y || ((x | y) << 1) == 0;
}
__device__ __forceinline__ bool same3(const double* a, const double* b) {
  return same(a[0], b[0]) && same(a[1], b[1]) && same(a[2], b[2]);
}
// g, or zero at or below eps (the skip of blade_vind_bywake, src/classdef.f90:1452-1466)
__device__ __forceinline__ double above_eps(double g) { return fabs(g) > kEps ? g : 0.0; }

// Lattice form of near-wake ring (b, i, j) (i the absolute row): edge k's weight
// (see vlm_bs.h).  Edge k of a ring is edge k ^ 2 of its neighbour on that side,
// run backwards; with the same end points and core radius the two filaments are
// one with the circulation difference, which edges 0 and 1 carry and their
// counterparts 2 and 3 leave out.
__device__ double lattice_weight(const Dims& d, const DevState& s, const double* nc, int b, int i, int j, int k,
                                 int rowNear) {
  const size_t r = ringI(d, b, i, j);
  const double G = above_eps(s.nGam[r]);
  const bool exists = k == 0 ? j > 0 : k == 1 ? i + 1 < d.NW : k == 2 ? j + 1 < d.ns : i > rowNear - 1;
  if (!exists) return G;
  const size_t o = k == 0 ? ringI(d, b, i, j - 1) : k == 1 ? r + 1 : k == 2 ? ringI(d, b, i, j + 1) : r - 1;
  const int kb = k ^ 2;  // the neighbour's edge
  const bool merged = same3(nc + 12 * o + 3 * ((kb + 1) & 3), nc + 12 * r + 3 * k) &&
                      same3(nc + 12 * o + 3 * kb, nc + 12 * r + 3 * ((k + 1) & 3)) &&
                      same(s.nRvc[4 * o + kb], s.nRvc[4 * r + k]);
  if (!merged) return G;
  return k < 2 ? G - above_eps(s.nGam[o]) : 0.0;
}

__device__ __forceinline__ bool same_bits(const double* a, const double* b, int n) {
  bool f = true;
  for (int k = 0; k < n; ++k) f &= __double_as_longlong(a[k]) == __double_as_longlong(b[k]);
  return f;
}
// What lane k of a ring's four finds it shares with its neighbours, bit for bit
// (k_lattice64): lane 3 corner 3 and edge 3 with the ring before (corners cb, radii
// vb), lane 0 corner 1 and edge 0 with the ring L before (ca, va); null: none.
__device__ __forceinline__ int shared_with(int k, const double* c, const double* v, const double* cb, const double* vb,
                                           const double* ca, const double* va) {
  if (k == 3 && cb && same_bits(c + 9, cb + 6, 3))
    return kShareC3 | (same_bits(c, cb + 3, 3) && same_bits(v + 3, vb + 1, 1) ? kShareE3 : 0);
  if (k == 0 && ca && same_bits(c + 3, ca + 6, 3))
    return kShareC1 | (same_bits(c, ca + 9, 3) && same_bits(v, va + 2, 1) ? kShareE0 : 0);
  return 0;
}

__global__ void __launch_bounds__(256) k_gather(Dims d, DevState s, const double* fr, const Group* groups, int ngroups,
                                                int nrec, int rowNear, int rowFar, int pred, float nearFactor, int L,
                                                int recBlocks, GatherTargets tg) {
  after_previous();
  if ((int)blockIdx.x >= recBlocks) {
    const int m = (blockIdx.x - recBlocks) * blockDim.x + threadIdx.x;
    if (m < tg.M)
      st3(tg.P + 3 * (size_t)m, tg.kind == 1 ? ld3(panRec(d, fr, m / d.npan, m % d.npan) + 12)
                                             : node_position(d, s, rowNear, rowFar, pred, m));
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x < 2 && tg.zero[threadIdx.x]) *tg.zero[threadIdx.x] = 0;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = q < 4 * nrec;
  const int t = live ? q >> 2 : 0, k = q & 3;
  int g = 0;
  while (g + 1 < ngroups && t >= groups[g + 1].rec_begin) ++g;
  const Group G = groups[g];
  const int l0 = t - G.rec_begin;
  const int b = G.blade;
  const double* corner = nullptr;  // the record's corners, or a single filament's ends
  double rv = 0.0, gam, W = 0.0;   // filament k's core radius, the circulation, edge k's weight
  int flags = 0, share = 0;
  if (G.kind == 0) {
    const int p = l0;
    corner = panRec(d, fr, b, p);
    rv = s.wRvc[4 * ((size_t)b * d.npan + p) + k];
    gam = s.wGam[(size_t)b * d.npan + p];
    W = gam;  // wing rings: no eps skip
    if (s.share) {
      const double* v = s.wRvc + 4 * ((size_t)b * d.npan + p);
      share = shared_with(k, corner, v, p > 0 ? panRec(d, fr, b, p - 1) : nullptr, v - 4, nullptr, nullptr);
    }
  } else {
    const int rowsN = d.NW - (rowNear - 1);
    const int nNear = rowsN * d.ns;
    const int hs = rowFar <= d.NF ? d.ns : 0;
    const int nFar = rowFar <= d.NF ? d.NF - rowFar + 1 : 0;
    const double* nc = pred ? s.nCP : s.nC;
    // a far-only group (pad[0] = 1) lists the far filaments alone, from the
    // pad[1]-th active one
    const int l = G.pad[0] ? l0 + nNear + hs + G.pad[1] : l0;
    if (l < nNear) {
      const int j = l / rowsN, i = rowNear - 1 + l % rowsN;
      const size_t r = ringI(d, b, i, j);
      corner = nc + 12 * r;
      rv = s.nRvc[4 * r + k];
      gam = s.nGam[r];
      flags = REC_SKIP;
      if (s.edgeW) W = lattice_weight(d, s, nc, b, i, j, k, rowNear);
      if (s.share) {
        const size_t a = j > 0 ? ringI(d, b, i, j - 1) : r;
        share = shared_with(k, corner, s.nRvc + 4 * r, i > rowNear - 1 ? nc + 12 * (r - 1) : nullptr, s.nRvc + 4 * r - 4,
                            j > 0 && rowsN == L ? nc + 12 * a : nullptr, s.nRvc + 4 * a);
      }
    } else if (l < nNear + hs) {
      // the horseshoe's closing filaments
      const size_t r = ringI(d, b, d.NW - 1, l - nNear);
      corner = nc + 12 * r + 3;
      rv = k ? 0.0 : s.nRvc[4 * r + 1];
      gam = -s.nGam[r];
      flags = REC_FIL;
      W = k ? 0.0 : gam;
    } else if (l >= nNear + hs + nFar) {
      // prescribed far wake (classdef.f90:1471-1476): single filaments
      const int i = l - nNear - hs - nFar;
      const size_t pb = (size_t)pred * d.nb + b;
      corner = s.pfC + (pb * kPresc + i) * 6;
      rv = k ? 0.0 : s.pfRvc[pb];
      gam = s.pfGam[pb];
      flags = REC_FIL | REC_SKIP;
      W = k ? 0.0 : above_eps(gam);
    } else {
      const size_t f = (size_t)b * d.NF + rowFar - 1 + (l - nNear - hs);
      corner = (pred ? s.fCP : s.fC) + 6 * f;
      rv = k ? 0.0 : s.fRvc[f];
      gam = s.fGam[f];
      flags = REC_FIL | REC_SKIP;
      W = k ? 0.0 : above_eps(gam);
    }
  }
  const bool fil = flags & REC_FIL;
  const d3 p = ld3(corner + 3 * (fil ? (k == 1 || k == 2 ? 1 : 0) : k));
  if (live) {
    double* R = s.rec64 + (size_t)t * kRec64;
    st3(R + 3 * k, fil && k >= 2 ? zero3() : p);
    R[12 + k] = rv;
    if (k == 0) R[16] = gam;
    if (k == 1) R[17] = (double)flags;
    if (s.edgeW) s.edgeW[4 * (size_t)t + k] = W;
  }
  if (s.share) {
    share |= __shfl_xor_sync(0xffffffffu, share, 1);
    share |= __shfl_xor_sync(0xffffffffu, share, 2);
    if (live && k == 0) s.share[t] = share;
  }
  if (s.rec32)
    pack_edge32(p, rv, gam, flags, s.edgeW != nullptr, W, k, nearFactor,
                live ? s.rec32 + (size_t)t * kRec32 : nullptr);
}

}  // namespace

void launch_gather(const Dims& d, const DevState& s, const double* frame, const Group* groups, int ngroups, int nrec,
                   int rowNear, int rowFar, bool pred, double nearFactor, int L, const GatherTargets& tg, cudaStream_t st) {
  const int rb = (int)(((long)nrec * 4 + 255) / 256), tb = tg.kind ? (tg.M + 255) / 256 : 0;
  if (rb + tb <= 0) return;
  count_launch();
  launch_next(k_gather, rb + tb, 256, 0, st, d, s, frame, groups, ngroups, nrec, rowNear, rowFar, pred ? 1 : 0,
              (float)nearFactor, L, rb, tg);
}

}  // namespace vlm
