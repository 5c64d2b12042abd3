// FP64 Biot-Savart partial sums in the reference's arithmetic, the chunk
// combiner, and the chunk-table builder.
//
// Compiled with -fmad=false: every multiply and add rounds separately, as in
// the oracle (built with -ffp-contract=off), so a chunked FP64 evaluation
// equals the oracle's evaluation with the same chunk size bit for bit.
#include <algorithm>
#include <atomic>

#include "launch.h"
#include "exact64.h"
#include "vlm_bs.h"
#include "vlm_math.h"

namespace vlm {

namespace {

// FP64 partial sums.  A warp's FP64 instruction holds its quarter of the SM
// for 64 cycles (half a lane a cycle), so the pair evaluations bound every
// shape here; a few warps on an SM fill the unit, and what a small shape lacks
// is quarters.  So the evaluations of a chunk are spread over threads and only
// its additions, which have to stay in record order, are serial: a block takes TT
// targets and evaluates a batch of S = threads / TT consecutive records of each at
// once into shared memory; 3 TT lanes, one for each (target, component), then add
// the S contributions in record order -- one to three warps, which take turns --
// while all go on with the next batch.  Each contribution and each addition is
// the reference's own, so the bits are those of one thread per target
// (blade_vind_bywing / blade_vind_bywake, src/classdef.f90:1342-1513).  The FP64
// pipe is busy for 90 % of k_rings64's cycles at 2^18 rings and 2048 targets and
// for 82 % of k_lattice64's at a 3-revolution hover wake.
//
// A near-wake sheet's rings are listed column by column (L rows each): ring
// r's corner 3 and edge 3 are ring r - 1's corner 2 and edge 1, its corner 1 and
// edge 0 ring r - L's corner 2 and edge 2.  An edge run backwards has exactly
// the negated velocity (every product and difference of vf_vind negates; only
// the sign of a zero may differ), so a ring whose neighbours are at hand costs
// one corner and two filaments, 111 FP64 instructions, instead of four and four,
// 211.  Corner 2's unit vector and edge 2 of the last L records stay in shared
// memory (48 bytes a target and row); share[r] says where the neighbours' hold
// bit for bit (a dissipated core, a row that just moved or the sheet's border
// breaks it, and a block's run of K chunks starts without neighbours), elsewhere
// the ring evaluates its own.
constexpr int kThreads64 = 128;          // rings one by one
constexpr int kThreadsLattice64 = 256;  // sheets: the wider block shares a column's buffer among more warps
constexpr int kMaxTT = 32;

// A record's flags and the reference's |gam| > eps, read from the words of the
// doubles: a conversion or a comparison would go through the FP64 unit.
__device__ __forceinline__ bool is_fil(const double* R) {
  const unsigned h = (unsigned)__double2hiint(R[17]);
  return h == 0x3ff00000u || h == 0x40080000u;  // 1 or 3
}
__device__ __forceinline__ bool skipped(const double* R) {
  const unsigned long long g = (unsigned long long)__double_as_longlong(R[16]) & 0x7fffffffffffffffull;
  const unsigned long long lo = 0x3cb0000000000001ull;  // the number after kEps = 2^-52
  return (unsigned)__double2hiint(R[17]) >= 0x40000000u && !(g - lo <= 0x7ff0000000000000ull - lo);
}
static_assert(REC_FIL == 1 && REC_SKIP == 2, "flag words");

__device__ __forceinline__ d3 contribution64(const exact64::Unit& u, d3 p, const double* __restrict__ R) {
  if (skipped(R)) return zero3();
  d3 v;
  if (is_fil(R)) {
    v = exact64::fil_vind(u, p, mk3(R[0], R[1], R[2]), mk3(R[3], R[4], R[5]), R[12]);
  } else {
    const d3 c[4] = {mk3(R[0], R[1], R[2]), mk3(R[3], R[4], R[5]), mk3(R[6], R[7], R[8]), mk3(R[9], R[10], R[11])};
    v = exact64::vr_vind(u, p, c, R + 12);
  }
  return exact64::mul(u, v, R[16]);
}

// The batch of n records from f whose contributions are in C added to the open
// chunk's sums acc in record order, one (component, target) a lane of the warps
// whose turn it is; q, qend: the open chunk and its end.
template <int NT>
__device__ __forceinline__ void add_batch64(const exact64::Unit& u, const double* C, double* acc, int turn, int lgTT,
                                            int f, int n, int q, int qe, int qend, const Chunk* __restrict__ chunks,
                                            int m0, int M, double* __restrict__ part) {
  const int TT = 1 << lgTT;
  const int lane = (threadIdx.x - 32 * (turn & (NT / 32 - 1))) & (NT - 1);
  if (lane >= 3 * TT) return;
  double a = acc[lane];
  for (int i = 0; i < n;) {
    const int e = min(n, qend - f);  // to the chunk's end
#pragma unroll 4
    for (; i < e; ++i) a = exact64::add(u, a, C[3 * TT * i + lane]);
    if (f + i == qend) {
      const int mk = m0 + (lane & (TT - 1));
      if (mk < M) part[((size_t)q * M + mk) * 3 + (lane >> lgTT)] = a;
      a = 0.0;
      if (++q < qe) qend += chunks[q].rec_count;
    }
  }
  acc[lane] = a;
}

// Grid: (target tiles) x (runs of K consecutive chunks).  lgTT = log2(TT).
__global__ void __launch_bounds__(kThreads64) k_rings64(const double* rec, const Chunk* chunks,
                                                       int nchunks, int K, const double* P, int M, int lgTT,
                                                       double* part) {
  after_previous();
  __shared__ double C[2][3 * kThreads64];  // contributions of two batches [s][component][t]
  __shared__ double acc[3 * kMaxTT];       // the open chunk's sums [component][t]
  const int TT = 1 << lgTT, S = kThreads64 >> lgTT;
  const exact64::Unit u = exact64::load_unit();
  const int t = threadIdx.x & (TT - 1), s = threadIdx.x >> lgTT;
  const int m0 = blockIdx.x * TT;
  const int m = min(m0 + t, M - 1);
  int q = blockIdx.y * K;
  const int qe = min(q + K, nchunks);
  const int r0 = chunks[q].rec_begin;
  const int r1 = chunks[qe - 1].rec_begin + chunks[qe - 1].rec_count;
  const d3 p = mk3(P[3 * (size_t)m], P[3 * (size_t)m + 1], P[3 * (size_t)m + 2]);
  if (threadIdx.x < 3 * TT) acc[threadIdx.x] = 0.0;
  int qend = r0 + chunks[q].rec_count;
  const int nb = (r1 - r0 + S - 1) / S;
  for (int b = 0; b <= nb; ++b) {
    const int r = r0 + b * S + s;
    if (r < r1) {
      const d3 v = contribution64(u, p, rec + (size_t)r * kRec64);
      double* c = C[b & 1] + 3 * TT * s + t;
      c[0] = v.x;
      c[TT] = v.y;
      c[2 * TT] = v.z;
    }
    if (b > 0) {
      const int f = r0 + (b - 1) * S, n = min(S, r1 - f);
      add_batch64<kThreads64>(u, C[(b - 1) & 1], acc, b, lgTT, f, n, q, qe, qend, chunks, m0, M, part);
      while (q < qe && qend <= f + n)
        if (++q < qe) qend += chunks[q].rec_count;
    }
    __syncthreads();
  }
}

// Between the first barrier of a batch and the second: corners 2 of the batch
// and the contributions of the one before; between the second and the next
// first: its edges and the additions of the one before.
__global__ void __launch_bounds__(kThreadsLattice64) k_lattice64(const double* rec, const int* share,
                                                         const Chunk* chunks, int nchunks, int K,
                                                         const double* P, int M, int lgTT, int L,
                                                         double* part) {
  after_previous();
  extern __shared__ double sm[];
  constexpr int NT = kThreadsLattice64;
  constexpr int B = 3 * NT;  // a batch's vectors in doubles, [s][component][t]
  const int TT = 1 << lgTT, S = NT >> lgTT;
  const int slots = L + S;
  double* acc = sm;                 // the open chunk's sums [component][t]
  double* C = acc + 3 * kMaxTT;     // contributions
  double* O = C + B;         // edges 0 and 3 of the rings that do not share them
  double* E1 = O + 2 * B;    // edge 1 of two batches
  double* U = E1 + 2 * B;    // corner 2's unit vector of the last records [slot][component][t]
  double* E2 = U + (size_t)3 * slots * TT;  // edge 2 of the last records
  const exact64::Unit u = exact64::load_unit();
  const int t = threadIdx.x & (TT - 1), s = threadIdx.x >> lgTT;
  const int m0 = blockIdx.x * TT;
  const int m = min(m0 + t, M - 1);
  int q = blockIdx.y * K;
  const int qe = min(q + K, nchunks);
  const int r0 = chunks[q].rec_begin;
  const int r1 = chunks[qe - 1].rec_begin + chunks[qe - 1].rec_count;
  const d3 p = mk3(P[3 * (size_t)m], P[3 * (size_t)m + 1], P[3 * (size_t)m + 2]);
  if (threadIdx.x < 3 * TT) acc[threadIdx.x] = 0.0;
  int qend = r0 + chunks[q].rec_count;
  auto put = [&](double* a, d3 v) {
    a[0] = v.x;
    a[TT] = v.y;
    a[2 * TT] = v.z;
  };
  auto take = [&](const double* a) { return mk3(a[0], a[TT], a[2 * TT]); };
  // what ring r shares with the rings of this run
  auto shared_bits = [&](int r) {
    int b = share[r];
    if (r - 1 < r0) b &= ~(kShareC3 | kShareE3);
    if (r - L < r0) b &= ~(kShareC1 | kShareE0);
    return b;
  };
  const int nb = (r1 - r0 + S - 1) / S;
  int slot = s, base = 0;  // this record's slot, and the first one's of the batch before
  for (int b = 0; b <= nb; ++b) {
    const int r = r0 + b * S + s, at = 3 * TT * s + t;
    const double* R = rec + (size_t)r * kRec64;
    const bool live = r < r1;
    const bool fil = live && is_fil(R);
    corner64 c2;
    if (live && !fil) {
      c2 = exact64::make_corner(u, p, mk3(R[6], R[7], R[8]));
      put(U + 3 * TT * slot + t, c2.u);
    }
    const int f = r0 + (b - 1) * S, n = min(S, r1 - f);  // the batch before
    if (b > 0) {
      for (int i = threadIdx.x; i < 3 * TT * n; i += NT) {
        const int si = (i >> lgTT) / 3, ri = f + si, ct = i - 3 * TT * si;
        const double* Ri = rec + (size_t)ri * kRec64;
        double v = O[i];
        if (!is_fil(Ri)) {
          const int sh = shared_bits(ri);
          int at2 = base + si;
          at2 -= at2 >= slots ? slots : 0;
          if (sh & kShareE0) v = -E2[3 * TT * (at2 >= L ? at2 - L : at2 - L + slots) + ct];
          const double* e1 = E1 + ((b - 1) & 1) * B;
          const double e3 = !(sh & kShareE3) ? O[B + i] : si ? -e1[i - 3 * TT] : -E1[(b & 1) * B + 3 * TT * (S - 1) + ct];
          v = exact64::add(u, exact64::add(u, exact64::add(u, v, e1[i]), E2[3 * TT * at2 + ct]), e3);
        }
        C[i] = skipped(Ri) ? 0.0 : exact64::mul(u, v, Ri[16]);
      }
      base += S;
      base -= base >= slots ? slots : 0;
    }
    __syncthreads();
    if (live) {
      if (fil) {
        put(O + at, exact64::fil_vind(u, p, mk3(R[0], R[1], R[2]), mk3(R[3], R[4], R[5]), R[12]));
      } else {
        const int sh = shared_bits(r);
        const d3 p1 = mk3(R[3], R[4], R[5]), p3 = mk3(R[9], R[10], R[11]);
        corner64 c1, c3;
        if (sh & kShareC1) {
          c1.r = exact64::sub(u, p, p1);
          c1.u = take(U + 3 * TT * (slot >= L ? slot - L : slot - L + slots) + t);
        } else {
          c1 = exact64::make_corner(u, p, p1);
        }
        put(E1 + (b & 1) * B + at, exact64::vf_vind(u, c1, c2, R[13]));
        if (sh & kShareC3) {
          c3.r = exact64::sub(u, p, p3);
          c3.u = take(U + 3 * TT * (slot ? slot - 1 : slots - 1) + t);
        } else {
          c3 = exact64::make_corner(u, p, p3);
        }
        put(E2 + 3 * TT * slot + t, exact64::vf_vind(u, c2, c3, R[14]));
        if ((sh & (kShareE0 | kShareE3)) != (kShareE0 | kShareE3)) {
          const corner64 c0 = exact64::make_corner(u, p, mk3(R[0], R[1], R[2]));
          if (!(sh & kShareE0)) put(O + at, exact64::vf_vind(u, c0, c1, R[12]));
          if (!(sh & kShareE3)) put(O + B + at, exact64::vf_vind(u, c3, c0, R[15]));
        }
      }
    }
    if (b > 0) {
      add_batch64<NT>(u, C, acc, b, lgTT, f, n, q, qe, qend, chunks, m0, M, part);
      while (q < qe && qend <= f + n)
        if (++q < qe) qend += chunks[q].rec_count;
    }
    slot += S;
    slot -= slot >= slots ? slots : 0;
    __syncthreads();
  }
}

// TT and K for M targets, nchunks chunks of nrec records in all and at most
// `largest` each, in sheets of L rows (0: rings one by one): the least modelled
// time on a device of `sms` SMs, a run taken as long as the longest (as long as the
// mean, a wing's short chunk beside its wake's made blocks of 8 targets of which
// the wake's were last to end: 124 us at 336 targets of a 40-step wing, now 77).
// A batch of a block that shares its quarters with w warps takes lat + w slope
// cycles (fitted to sweeps over TT and K from 52 to 60000 targets and 52 to 12480
// records; slope is its FP64 instructions, lat the chain of one evaluation),
// a run's first column of a sheet's edges a half more, and an ordered addition
// 90 in each warp whose turn it is.  Few targets and chunks get one target a
// block (a wing's 52 rings at 52 points: 52 blocks whose threads take a record
// each, 18 us; 906 us in one block of a thread per target), many get 4 to 16.
struct Tile64 {
  int lgTT = 0, K = 1;
};
constexpr size_t kSmemPerSm64 = 227 * 1024;
inline size_t lattice_smem64(int lgTT, int L) {
  const int TT = 1 << lgTT, nt = kThreadsLattice64;
  return sizeof(double) * (3 * kMaxTT + (size_t)15 * nt + (size_t)6 * TT * (L + nt / TT));
}
Tile64 pick_tile64(int M, int nchunks, int64_t nrec, int largest, int L, int sms) {
  const int nt = L > 0 ? kThreadsLattice64 : kThreads64;
  const double wb = nt / 128;
  double best = 0.0;
  Tile64 T;
  for (int lg = 0; (1 << lg) <= kMaxTT; ++lg) {
    const int TT = 1 << lg, S = nt / TT;
    const double tiles = (double)(((int64_t)M + TT - 1) / TT);
    int bps = 5;  // by their registers
    if (L > 0) bps = std::min<int>(2, (int)(kSmemPerSm64 / (lattice_smem64(lg, L) + 1024)));
    if (bps < 1) break;
    for (int k = 1;; k *= 2) {
      // a run's records: the longest, which is last to end
      const double runs = (nchunks + k - 1) / k, recs = (double)std::min<int64_t>(nrec, (int64_t)k * largest);
      const double batches = std::ceil(recs / S) + 0.3;
      const double lat = L > 0 ? 7700 : 11500, slope = L > 0 ? 8000 + 3200 * std::min(1.0, L / recs) : 13600;
      const double add = 90.0 * std::min<double>(S, recs);
      const double X = tiles * runs / sms;  // blocks per SM
      double t;
      if (X <= bps) t = batches * (lat + slope * wb * std::ceil(X) + add);
      else t = (tiles * (nrec / (double)S + 0.8 * runs) / sms / bps + 0.15 * batches) * (lat + slope * wb * bps + add);
      if (best == 0.0 || t < best * 0.999) {
        best = t;
        T.lgTT = lg;
        T.K = k;
      }
      if (k >= nchunks || k >= 32) break;
    }
  }
  return T;
}

// FP64: each group's partials in chunk order, one component of a target a
// thread, loads 16 at a time (a collocation-point evaluation has few targets
// and hundreds of chunks).
__device__ __forceinline__ double group_sum(const double* part, int M, const Group& g, size_t mc) {
  const size_t stride = 3 * (size_t)M;
  double s = 0.0;
  const double* p = part + g.chunk_begin * stride + mc;
  int q = 0;
  constexpr int kB = 16;
  for (; q + kB <= g.chunk_count; q += kB, p += kB * stride) {
    double buf[kB];
#pragma unroll
    for (int i = 0; i < kB; ++i) buf[i] = p[i * stride];
#pragma unroll
    for (int i = 0; i < kB; ++i) s = s + buf[i];
  }
  for (; q < g.chunk_count; ++q, p += stride) s = s + p[0];
  return s;
}

// mode 0 (wake nodes): out = 0 + (wing + wake); 1: wake; 2: wing + wake.
__global__ void k_combine(const double* part, int M, const Group* groups, int ngroups, int mode, double* out) {
  after_previous();
  const size_t mc = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (mc >= 3 * (size_t)M) return;
  double wing = 0.0, wake = 0.0;
  for (int g = 0; g < ngroups; ++g) {
    const Group gr = groups[g];
    const double s = group_sum(part, M, gr, mc);
    if (gr.kind == 0) wing = wing + s;
    else wake = wake + s;
  }
  out[mc] = mode == 0 ? 0.0 + (wing + wake) : mode == 1 ? wake : wing + wake;
}

// Coupled rotors: the groups carry the index of the sum they belong to
// (Group::term, non-decreasing).  mode 0 (wake nodes, src/main.f90:808-827):
// v = 0, then v = v + (wing_t + wake_t) for every term in turn, one term per
// source rotor (libCommon.f90:114-211 adds a rotor's wing and wake);
// out[m] = v.  mode 3 (collocation points, src/main.f90:549-561):
// out[t][m] = 0 + the term's groups in order, one per-rotor wake or wing
// sum each, which the RHS adds to velCP in turn.  With a single term, mode 0
// equals k_combine's mode 0 bit for bit.
__global__ void k_combine_terms(const double* part, int M, const Group* groups, int ngroups, int mode, double* out) {
  after_previous();
  const size_t mc = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (mc >= 3 * (size_t)M) return;
  double v = 0.0, wing = 0.0, wake = 0.0, ts = 0.0;
  int t = groups[0].term;
  auto done = [&]() {
    if (mode == 0) v = v + (wing + wake);
    else out[3 * (size_t)M * t + mc] = ts;
    wing = wake = ts = 0.0;
  };
  for (int g = 0; g < ngroups; ++g) {
    const Group gr = groups[g];
    if (gr.term != t) {
      done();
      t = gr.term;
    }
    const double s = group_sum(part, M, gr, mc);
    if (mode != 0) ts = ts + s;
    else if (gr.kind == 0) wing = wing + s;
    else wake = wake + s;
  }
  done();
  if (mode == 0) out[mc] = v;
}

// FP32 paths, whose summation order is free: the partials of a target
// component, whatever their group, over G lanes (a power of two <= 32; lane l
// adds chunks l, l + G, ...), then a butterfly; the tree has a fixed shape, so
// the result is reproducible run to run.  nacc: the near field's fixed-point
// corrections of the same partials, zeroed on the way and added as the integers
// that they are, with one conversion at the end (those of 64 and more, of
// which a lane's few thousand could overflow, one by one): conversions and
// additions run on the FP64 unit, 16 cycles a warp and SM, and bound the kernel.
// Group by group, each with its own butterfly and a conversion a partial, 13500
// targets of 24 chunks took 33 us, now 15; 48 of 300 took 12, now 7.  mode 3: term
// blockIdx.y's groups alone, into its part of out; mode 1 leaves the wings' chunks out.
template <bool ADD>
__global__ void __launch_bounds__(256) k_combine_tree(const double* part, long long* nacc, int M, const Group* groups,
                                                      int ngroups, int mode, int G, double* out) {
  after_previous();
  const size_t gt = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t mc = gt / G, stride = 3 * (size_t)M;
  const int l = (int)(gt % G);
  const bool live = mc < stride;  // dead lanes still take part in the shuffles
  double s = 0.0;
  long long sum = 0;
  auto range = [&](int a, int b, bool use) {
    constexpr int kB = 4;
    for (int q = a + l; q < b; q += kB * G) {
      double p[kB];
      long long n[kB];
#pragma unroll
      for (int i = 0; i < kB; ++i) {
        const bool in = q + i * G < b;
        p[i] = in && use ? part[(q + i * G) * stride + mc] : 0.0;
        n[i] = in && nacc ? nacc[(q + i * G) * stride + mc] : 0;
      }
#pragma unroll
      for (int i = 0; i < kB; ++i) {
        if (q + i * G < b) s = s + p[i];
        if (n[i] != 0) {
          nacc[(q + i * G) * stride + mc] = 0;
          if (!use) continue;
          constexpr long long kBig = (long long)1 << 50;
          if ((unsigned long long)(n[i] + kBig) < 2ull * kBig) sum += n[i];
          else s = s + (double)n[i] * (1.0 / kNearScale);
        }
      }
    }
  };
  if (live) {
    int g0 = 0, g1 = ngroups;
    if (mode == 3) {
      while (g0 < ngroups && groups[g0].term < (int)blockIdx.y) ++g0;
      g1 = g0;
      while (g1 < ngroups && groups[g1].term == (int)blockIdx.y) ++g1;
    }
    if (mode == 1) {
      for (int g = g0; g < g1; ++g)
        range(groups[g].chunk_begin, groups[g].chunk_begin + groups[g].chunk_count, groups[g].kind != 0);
    } else if (g0 < g1) {
      range(groups[g0].chunk_begin, groups[g1 - 1].chunk_begin + groups[g1 - 1].chunk_count, true);
    }
  }
  if (sum != 0) s = s + (double)sum * (1.0 / kNearScale);
  for (int o = G >> 1; o > 0; o >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, o, G);
  if (!live || l != 0) return;
  if (mode == 3) out += stride * blockIdx.y;
  out[mc] = ADD ? out[mc] + s : s;
}

// lanes per (target, component): about 8 chunk partials each, at most a warp
inline int tree_lanes(int nchunks) {
  int G = 1;
  while (G < 32 && G * 8 < nchunks) G <<= 1;
  return G;
}

__global__ void k_rings_to_rec64(const double* corners, const double* rvc,
                                 const double* gam, int64_t N, double* rec) {
  after_previous();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= N) return;
  double* R = rec + n * kRec64;
  for (int k = 0; k < 12; ++k) R[k] = corners[n * 12 + k];
  for (int k = 0; k < 4; ++k) R[12 + k] = rvc[n * 4 + k];
  R[16] = gam[n];
  R[17] = 0.0;
}

// Single filaments fc1 -> fc2 (vf_vind, src/classdef.f90:476-503) as
// REC_FIL records; no |gam| skip (gridgen sums every filament,
// src/gridgen.f90:128-136).
__global__ void k_fils_to_rec64(const double* fc, const double* rvc,
                                const double* gam, int64_t N, double* rec) {
  after_previous();
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= N) return;
  double* R = rec + n * kRec64;
  for (int k = 0; k < 6; ++k) R[k] = fc[n * 6 + k];
  for (int k = 6; k < 12; ++k) R[k] = 0.0;
  R[12] = rvc[n];
  R[13] = R[14] = R[15] = 0.0;
  R[16] = gam[n];
  R[17] = (double)REC_FIL;
}

}  // namespace

static std::atomic<long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void count_launches(long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long launch_count() { return g_launches.load(); }

int build_chunks(Group* groups, int ngroups, int chunk_size, Chunk* chunks, int cap) {
  int nq = 0;
  for (int g = 0; g < ngroups; ++g) {
    Group& G = groups[g];
    G.chunk_begin = nq;
    G.chunk_count = 0;
    if (G.rec_count <= 0) continue;
    const int C = chunk_size > 0 ? chunk_size : G.rec_count;
    for (int r = 0; r < G.rec_count; r += C) {
      if (nq >= cap) return -1;
      chunks[nq].rec_begin = G.rec_begin + r;
      chunks[nq].rec_count = std::min(C, G.rec_count - r);
      ++nq;
      ++G.chunk_count;
    }
  }
  return nq;
}

namespace {
dim3 grid64(const Tile64& T, int M, int nchunks, int& K) {
  K = std::max(T.K, (nchunks + 65534) / 65535);  // the grid's second dimension ends at 65535
  return dim3((unsigned)(((int64_t)M + (1 << T.lgTT) - 1) >> T.lgTT), (unsigned)((nchunks + K - 1) / K));
}
// the dynamic shared-memory opt-in is per device; set it once on each
void lattice_attr64() {
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && attr[dev].load(std::memory_order_acquire)) return;
  cudaFuncSetAttribute(k_lattice64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerSm64);
  if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
}
void launch_rings64(const Tile64& T, const double* rec, const Chunk* chunks, int nchunks, const double* P, int M,
                    double* part, cudaStream_t s) {
  int K = 1;
  const dim3 grid = grid64(T, M, nchunks, K);
  launch_next(k_rings64, grid, kThreads64, 0, s, rec, chunks, nchunks, K, P, M, T.lgTT, part);
}
void launch_lattice64(const Tile64& T, const double* rec, const int* share, const Chunk* chunks, int nchunks, int L,
                      const double* P, int M, double* part, cudaStream_t s) {
  int K = 1;
  const dim3 grid = grid64(T, M, nchunks, K);
  launch_next(k_lattice64, grid, kThreadsLattice64, lattice_smem64(T.lgTT, L), s, rec, share, chunks, nchunks, K, P, M,
              T.lgTT, L, part);
}
}  // namespace

void launch_partial64(const double* rec, const Chunk* chunks, int nchunks, int64_t nrec, int largest, const double* P, int M,
                      double* part, cudaStream_t s) {
  if (M <= 0 || nchunks <= 0) return;
  count_launch();
  launch_rings64(pick_tile64(M, nchunks, nrec, largest, 0, device_sm_count()), rec, chunks, nchunks, P, M, part, s);
}

void launch_partial64_lattice(const double* rec, const Chunk* chunks, int nchunks, int nrec, int largest, int L,
                              const int* share, const double* P, int M, double* part, cudaStream_t s) {
  // A sheet too tall for shared memory even with one target a block (above 3909
  // rows) has no room for a column's edges.  Sheets of 8 stations, ns a ring and
  // target: 0.39 at 1488 rows, where an SM still holds two blocks of one target,
  // 0.45 at 1489, where it holds one, 0.60 at 2500, 0.64 at 3909, and 0.37 ring
  // by ring at 3910: by time the line would lie at 1488.
  if (L <= 0 || lattice_smem64(0, L) + 1024 > kSmemPerSm64) {
    launch_partial64(rec, chunks, nchunks, nrec, largest, P, M, part, s);
    return;
  }
  if (M <= 0 || nchunks <= 0) return;
  lattice_attr64();
  count_launch();
  launch_lattice64(pick_tile64(M, nchunks, nrec, largest, L, device_sm_count()), rec, share, chunks, nchunks, L, P, M,
                   part, s);
}

void launch_combine(const double* part, int M, const Group* groups, int ngroups, int mode, double* out,
                    cudaStream_t s) {
  if (M <= 0) return;
  count_launch();
  launch_next(k_combine, (unsigned)((3 * (size_t)M + 127) / 128), 128, 0, s, part, M, groups, ngroups, mode, out);
}

void launch_combine_unordered(const double* part, long long* nacc, int M, const Group* groups, int ngroups,
                              int nchunks, int mode, double* out, cudaStream_t s, bool add) {
  if (M <= 0) return;
  const int G = tree_lanes(nchunks);
  const unsigned blocks = (unsigned)((3 * (size_t)M * G + 255) / 256);
  count_launch();
  if (add) launch_next(k_combine_tree<true>, blocks, 256, 0, s, part, nacc, M, groups, ngroups, mode, G, out);
  else launch_next(k_combine_tree<false>, blocks, 256, 0, s, part, nacc, M, groups, ngroups, mode, G, out);
}

void launch_combine_terms(const double* part, long long* nacc, int M, const Group* groups, int ngroups,
                          int nchunks, int nterms, int mode, bool ordered, double* out, cudaStream_t s) {
  if (M <= 0 || ngroups <= 0) return;
  count_launch();
  if (ordered) {
    launch_next(k_combine_terms, (unsigned)((3 * (size_t)M + 127) / 128), 128, 0, s, part, M, groups, ngroups, mode, out);
    return;
  }
  const int per = mode == 3 ? nterms : 1, G = tree_lanes((nchunks + per - 1) / per);
  launch_next(k_combine_tree<false>, dim3((unsigned)((3 * (size_t)M * G + 255) / 256), per), 256, 0, s, part, nacc, M,
              groups, ngroups, mode, G, out);
}

void launch_fils_to_rec64(const double* fc, const double* rvc, const double* gam, int64_t N, double* rec,
                          cudaStream_t s) {
  if (N <= 0) return;
  count_launch();
  launch_next(k_fils_to_rec64, (unsigned)((N + 255) / 256), 256, 0, s, fc, rvc, gam, N, rec);
}

void launch_rings_to_rec64(const double* corners, const double* rvc, const double* gam, int64_t N, double* rec,
                           cudaStream_t s) {
  if (N <= 0) return;
  count_launch();
  launch_next(k_rings_to_rec64, (unsigned)((N + 255) / 256), 256, 0, s, corners, rvc, gam, N, rec);
}

}  // namespace vlm
