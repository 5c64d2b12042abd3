// Incremental predicted-wake evaluation (FP32 precisions).
//
// The predictor of the reference's predictor-corrector and Adams-Moulton
// schemes (fdSchemeSwitch 1, 3, 4, 5: src/main.f90:844-1406) moves a small
// part of the wake -- its 'P' convection loops `do i = 1, rowNear, nNwake`
// and so visits the first near-wake row only (src/classdef.f90:1549-1575):
// the predicted wake differs from the current one in a few node rows and the
// far-wake filaments.  Every source record and every target point that did not
// move gives the same FP32 pair in both evaluations, so the predicted-wake
// velocity at an unmoved target is the current-wake velocity plus the sum of
// (new - old) over the moved records, and only the moved targets need the full
// sum.  These kernels find the moved records and targets by comparing the two
// gathered record sets and target sets bit by bit, compact them in index order
// (a deterministic order, so that a replayed step gives the same bits) into
// fixed-capacity buffers padded with inert records, and merge the results.
#include <cuda_runtime.h>

#include <algorithm>

#include "launch.h"
#include "vlm_bs.h"

namespace vlm {
namespace {

// small tiles: a record is 18 + 4 doubles, read by one thread, and a few
// hundred blocks keep every SM busy on a 25k-record set
constexpr int kDiffThreads = 128;
constexpr int kDiffItems = 2;  // items per thread per block tile
constexpr int kDiffTile = kDiffThreads * kDiffItems;

// item i of N doubles differs between the two sets
template <int N>
__device__ __forceinline__ bool item_differs(const double* a, const double* b, int i) {
  unsigned long long x = 0;
#pragma unroll
  for (int k = 0; k < N; ++k)
    x |= (unsigned long long)__double_as_longlong(a[(size_t)i * N + k]) ^
         (unsigned long long)__double_as_longlong(b[(size_t)i * N + k]);
  return x != 0;
}
// record i differs: its doubles, or its 4 edge weights when the sets carry them
__device__ __forceinline__ bool record_differs(const double* a, const double* b, const double* ea, const double* eb, int i) {
  const bool f = item_differs<kRec64>(a, b, i);
  return ea ? f | item_differs<4>(ea, eb, i) : f;
}

// exclusive prefix of f over the block's threads in thread order; *total =
// the block's count.  Every thread of the block calls it.
__device__ __forceinline__ int block_prefix(bool f, int* warpTot, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, f);
  if (lane == 0) warpTot[w] = __popc(b);
  __syncthreads();
  int before = 0, tot = 0;
  for (int k = 0; k < kDiffThreads / 32; ++k) {
    const int c = warpTot[k];
    if (k < w) before += c;
    tot += c;
  }
  __syncthreads();  // warpTot is reused by the next call
  *total = tot;
  return before + __popc(b & ((1u << lane) - 1u));
}

// Two sets of items compared in one launch: records (with their edge weights, or
// none) and targets.
struct DiffSet {
  const double *a, *b, *ea, *eb;
  int n, blocks;
  int *blockCount, *total;
};

// per block tile of kDiffTile items: the number that changed (the records' tiles
// first).  All of an item's words are compared, in loads that do not wait for one
// another; leaving at the first difference made a chain of them (the counts and
// scans of a hover step's two sets, four launches: 14 us, now two of 6).
__global__ void __launch_bounds__(kDiffThreads) k_diff_count(DiffSet rec, DiffSet tgt) {
  after_previous();
  __shared__ int warpTot[kDiffThreads / 32];
  const bool isRec = (int)blockIdx.x < rec.blocks;
  const int block = isRec ? blockIdx.x : blockIdx.x - rec.blocks;
  int cnt = 0;
  for (int u = 0; u < kDiffItems; ++u) {
    const int i = block * kDiffTile + u * kDiffThreads + threadIdx.x;
    bool f = false;
    if (isRec) f = i < rec.n && record_differs(rec.a, rec.b, rec.ea, rec.eb, i);
    else f = i < tgt.n && item_differs<3>(tgt.a, tgt.b, i);
    int tot = 0;
    block_prefix(f, warpTot, &tot);
    cnt += tot;
  }
  if (threadIdx.x == 0) (isRec ? rec : tgt).blockCount[block] = cnt;
}

// exclusive scan of the block counts in place (block 0 the records', 1 the targets'); *total = their sum
__global__ void __launch_bounds__(kDiffThreads) k_diff_scan(DiffSet rec, DiffSet tgt) {
  after_previous();
  __shared__ int sh[kDiffThreads];
  int* blockCount = blockIdx.x == 0 ? rec.blockCount : tgt.blockCount;
  const int nb = blockIdx.x == 0 ? rec.blocks : tgt.blocks;
  int carry = 0;
  for (int base = 0; base < nb; base += kDiffThreads) {
    const int i = base + threadIdx.x;
    const int v = i < nb ? blockCount[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < kDiffThreads; off <<= 1) {
      const int t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    const int incl = sh[threadIdx.x];
    if (i < nb) blockCount[i] = carry + incl - v;
    carry += sh[kDiffThreads - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) *(blockIdx.x == 0 ? rec.total : tgt.total) = carry;
}

// The delta record set: changed record r (o-th in index order) -> slot 2o its
// predicted version (+), slot 2o + 1 its current version with the circulation
// negated (-): the edge weights when the sets carry them, else the record's
// circulation.  Slots from 2 min(total, half) to cap are inert: a copy of
// predicted record 0 with no circulation on any filament (lattice edge weights
// 0; or circulation 0 with the skip flag), which the FP32 packer turns into a
// record of zero weights and no near field.  More changed records than half
// the capacity: ctl = 5 (the step's result is then wrong and reported).
__global__ void __launch_bounds__(kDiffThreads)
    k_delta_records(const double* recP, const double* recC, const double* ewP,
                    const double* ewC, int nrec, const int* blockOff,
                    const int* total, double* dRec, double* dEw, int cap,
                    int* ctl) {
  after_previous();
  __shared__ int warpTot[kDiffThreads / 32];
  const int half = cap / 2;
  int off = blockOff[blockIdx.x];
  const int base = blockIdx.x * kDiffTile;
  for (int u = 0; u < kDiffItems; ++u) {
    const int r = base + u * kDiffThreads + threadIdx.x;
    const bool f = r < nrec && record_differs(recP, recC, ewP, ewC, r);
    int tot = 0;
    const int p = block_prefix(f, warpTot, &tot);
    const int o = off + p;
    if (f && o < half) {
      const double* P = recP + (size_t)r * kRec64;
      const double* C = recC + (size_t)r * kRec64;
      double* dn = dRec + (size_t)(2 * o) * kRec64;
      double* dd = dn + kRec64;
      for (int k = 0; k < kRec64; ++k) {
        dn[k] = P[k];
        dd[k] = C[k];
      }
      if (ewP) {
        for (int k = 0; k < 4; ++k) {
          dEw[4 * (size_t)(2 * o) + k] = ewP[4 * (size_t)r + k];
          dEw[4 * (size_t)(2 * o + 1) + k] = -ewC[4 * (size_t)r + k];
        }
      } else {
        dd[16] = -C[16];
      }
    }
    off += tot;
  }
  // inert padding, grid-stride over the whole capacity
  const int n = *total;
  const int used = 2 * min(n, half);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
    if (i < used) continue;
    double* dn = dRec + (size_t)i * kRec64;
    for (int k = 0; k < kRec64; ++k) dn[k] = recP[k];
    if (ewP) {
      for (int k = 0; k < 4; ++k) dEw[4 * (size_t)i + k] = 0.0;
    } else {
      dn[16] = 0.0;
      dn[17] = (double)((int)recP[17] | REC_SKIP);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > half) atomicCAS(ctl, 0, 5);
}

// The moved targets: o-th moved target (index order) -> idx[o], pos[o];
// slots from min(total, cap) to cap get target 0's position (their results are
// not used).  More than cap: ctl = 5.
__global__ void __launch_bounds__(kDiffThreads)
    k_moved_targets(const double* tP, const double* tC, int M,
                    const int* blockOff, const int* total, int* idx,
                    double* pos, int cap, int* ctl) {
  after_previous();
  __shared__ int warpTot[kDiffThreads / 32];
  int off = blockOff[blockIdx.x];
  const int base = blockIdx.x * kDiffTile;
  for (int u = 0; u < kDiffItems; ++u) {
    const int m = base + u * kDiffThreads + threadIdx.x;
    const bool f = m < M && item_differs<3>(tP, tC, m);
    int tot = 0;
    const int p = block_prefix(f, warpTot, &tot);
    const int o = off + p;
    if (f && o < cap) {
      idx[o] = m;
      for (int k = 0; k < 3; ++k) pos[3 * (size_t)o + k] = tP[3 * (size_t)m + k];
    }
    off += tot;
  }
  const int n = *total;
  const int used = min(n, cap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
    if (i < used) continue;
    for (int k = 0; k < 3; ++k) pos[3 * (size_t)i + k] = tP[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > cap) atomicCAS(ctl, 0, 5);
}

// also passes the moved targets' evaluation's error code on to the step's
__global__ void k_incr_put(double* out, const int* idx, const double* v,
                           const int* total, int cap, const int* subCtl,
                           int* ctl) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && subCtl[0] != 0) atomicCAS(ctl, 0, subCtl[0]);
  if (i >= min(*total, cap)) return;
  const int m = idx[i];
  for (int k = 0; k < 3; ++k) out[3 * (size_t)m + k] = v[3 * (size_t)i + k];
}

inline int diff_blocks(int n) { return (n + kDiffTile - 1) / kDiffTile; }

}  // namespace

int incr_diff_blocks(int n) { return n > 0 ? diff_blocks(n) : 0; }

void launch_diff_count(const double* recA, const double* recB, const double* ea, const double* eb, int nrec, int* blockR,
                       int* totalR, const double* tA, const double* tB, int M, int* blockT, int* totalT, cudaStream_t s) {
  const DiffSet rec{recA, recB, ea, eb, nrec, incr_diff_blocks(nrec), blockR, totalR};
  const DiffSet tgt{tA, tB, nullptr, nullptr, M, incr_diff_blocks(M), blockT, totalT};
  if (rec.blocks + tgt.blocks > 0) {
    count_launch();
    launch_next(k_diff_count, rec.blocks + tgt.blocks, kDiffThreads, 0, s, rec, tgt);
  }
  count_launch();
  launch_next(k_diff_scan, 2, kDiffThreads, 0, s, rec, tgt);
}

void launch_delta_records(const double* recP, const double* recC, const double* ewP, const double* ewC, int nrec,
                          const int* blockOff, const int* total, double* dRec, double* dEw, int cap, int* ctl,
                          cudaStream_t s) {
  if (nrec <= 0 || cap <= 0) return;
  count_launch();
  launch_next(k_delta_records, diff_blocks(nrec), kDiffThreads, 0, s, recP, recC, ewP, ewC, nrec, blockOff, total, dRec, dEw,
                                                            cap, ctl);
}

void launch_moved_targets(const double* tP, const double* tC, int M, const int* blockOff, const int* total, int* idx,
                          double* pos, int cap, int* ctl, cudaStream_t s) {
  if (M <= 0 || cap <= 0) return;
  count_launch();
  launch_next(k_moved_targets, diff_blocks(M), kDiffThreads, 0, s, tP, tC, M, blockOff, total, idx, pos, cap, ctl);
}

void launch_incr_merge(double* out, const int* idx, const double* moved, const int* total, int cap, const int* subCtl,
                       int* ctl, cudaStream_t s) {
  count_launch();
  launch_next(k_incr_put, (std::max(cap, 1) + 255) / 256, 256, 0, s, out, idx, moved, total, cap, subCtl, ctl);
}

}  // namespace vlm
