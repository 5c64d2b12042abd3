// LU factors and the explicit inverse of the AIC matrix (src/libMath.f90:48-122:
// inv2), in FP64 with the reference's operations in its order, and in FP32 for
// the refined solve.  Compiled with -fmad=false.
//
// LU with partial pivoting (first index of the largest magnitude), right-looking
// in panels of up to 16 columns: one block factors a panel in shared memory, one
// kernel applies its row interchanges to the other columns and solves for the
// panel's rows of U, one updates the trailing matrix.  Every element is updated by
// k = 0, 1, ... in turn as in the unblocked loop, so the bits are the same.  A
// column of 300 rows costs its panel about 2 us (two barriers, a division, 16
// updates on one SM's FP64 unit); the unblocked loop in one block took 21 us.
#include <math.h>

#include <algorithm>
#include <atomic>

#include "launch.h"
#include "exact64.h"
#include "vlm_math.h"
#include "vlm_solver.h"

namespace vlm {

namespace {

constexpr int kPanel = 16;
constexpr int kPanelThreads = 512;
constexpr size_t kSmemMax = 226 * 1024;

// a - b c, as the reference rounds it in FP64 and fused in FP32
__device__ __forceinline__ double sub_mul(double a, double b, double c) { return a - b * c; }
__device__ __forceinline__ float sub_mul(float a, float b, float c) { return fmaf(-b, c, a); }
// |a| as an integer that orders like it (a comparison of doubles takes the FP64
// unit), -1 for NaN, which no comparison prefers
__device__ __forceinline__ long long mag(double a) {
  const long long b = __double_as_longlong(a) & 0x7fffffffffffffffll;
  return b > 0x7ff0000000000000ll ? -1 : b;
}
__device__ __forceinline__ int mag(float a) {
  const int b = __float_as_int(a) & 0x7fffffff;
  return b > 0x7f800000 ? -1 : b;
}
template <class T>
struct Mag {
  typedef long long type;
};
template <>
struct Mag<float> {
  typedef int type;
};
// one divisor for a column's rows
struct ByDouble {
  double d;
  exact64::Root r;
  uint64_t Z;
  bool fast;
  __device__ explicit ByDouble(double x) : d(x), fast(exact64::divisor_in_range(x)) {
    if (fast) r = exact64::divisor_of(x), Z = exact64::reciprocal(r);
  }
  __device__ double operator()(double a) const {
    return fast && exact64::div_in_range(a) ? exact64::with_sign(exact64::divide(a, r, Z), d) : a / d;
  }
};
struct ByFloat {
  float d;
  __device__ explicit ByFloat(float x) : d(x) {}
  __device__ float operator()(float a) const { return a / d; }
};
__device__ __forceinline__ ByDouble by(double d) { return ByDouble(d); }
__device__ __forceinline__ ByFloat by(float d) { return ByFloat(d); }

template <class T>
__global__ void k_lu_copy(const double* A, T* LU, size_t n2) {
  after_previous();
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n2) LU[i] = (T)A[i];
}

// The interchanges of a panel as a permutation: row dst[i] takes row src[i], i < count.
struct Perm {
  int count, dst[2 * kPanel], src[2 * kPanel];
};

// Columns k0 .. k0 + nb - 1, rows k0 .. n - 1.  A thread keeps to its rows: it
// divides, updates the row's later columns and has the next column's candidates
// at hand; the block meets twice a column, for the pivot and after the swap.
template <class T>
__global__ void __launch_bounds__(kPanelThreads) k_lu_panel(T* A, int n, int k0, int nb,
                                                           int* piv, int* err,
                                                           Perm* perm) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  T* p = reinterpret_cast<T*>(smem);  // [column][row - k0]
  typedef typename Mag<T>::type MagT;
  __shared__ MagT wv[kPanelThreads / 32];
  __shared__ int wi[kPanelThreads / 32];
  __shared__ int pivots[kPanel];
  const int m = n - k0, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = 0; c < nb; ++c)
    for (int i = threadIdx.x; i < m; i += kPanelThreads) p[(size_t)c * m + i] = A[(size_t)(k0 + c) * n + k0 + i];
  MagT bv = -1;
  int bi = m;
  for (int i = threadIdx.x; i < m; i += kPanelThreads) {
    const MagT v = mag(p[i]);
    if (v > bv) bv = v, bi = i;  // a thread's rows come in order: the first of equals stays
  }
  __syncthreads();
  for (int c = 0; c < nb; ++c) {
    for (int o = 16; o > 0; o >>= 1) {
      const MagT v = __shfl_xor_sync(0xffffffffu, bv, o);
      const int i = __shfl_xor_sync(0xffffffffu, bi, o);
      if (v > bv || (v == bv && i < bi)) bv = v, bi = i;
    }
    if (lane == 0) wv[warp] = bv, wi[warp] = bi;
    __syncthreads();
    bv = lane < kPanelThreads / 32 ? wv[lane] : (MagT)-1;
    bi = lane < kPanelThreads / 32 ? wi[lane] : m;
    for (int o = 16; o > 0; o >>= 1) {
      const MagT v = __shfl_xor_sync(0xffffffffu, bv, o);
      const int i = __shfl_xor_sync(0xffffffffu, bi, o);
      if (v > bv || (v == bv && i < bi)) bv = v, bi = i;
    }
    const int r = bi < m ? bi : c;  // no candidate: a column of NaN
    if (threadIdx.x < nb && r != c) {
      T* q = p + (size_t)threadIdx.x * m;
      const T t = q[c];
      q[c] = q[r];
      q[r] = t;
    }
    if (threadIdx.x == 0) {
      pivots[c] = r;
      piv[k0 + c] = k0 + r;
    }
    __syncthreads();
    const T akk = p[(size_t)c * m + c];
    if (threadIdx.x == 0 && akk == (T)0 && err) atomicExch(err, 10);
    const auto over = by(akk);
    bv = -1;
    bi = m;
    for (int i = threadIdx.x; i < m; i += kPanelThreads) {
      if (i <= c) continue;
      const T l = over(p[(size_t)c * m + i]);
      p[(size_t)c * m + i] = l;
      for (int j = c + 1; j < nb; ++j) {
        const T a = sub_mul(p[(size_t)j * m + i], l, p[(size_t)j * m + c]);
        p[(size_t)j * m + i] = a;
        if (j == c + 1) {
          const MagT v = mag(a);
          if (v > bv) bv = v, bi = i;
        }
      }
    }
  }
  __syncthreads();
  for (int c = 0; c < nb; ++c)
    for (int i = threadIdx.x; i < m; i += kPanelThreads) A[(size_t)(k0 + c) * n + k0 + i] = p[(size_t)c * m + i];
  if (threadIdx.x == kPanelThreads - 1) {
    // the interchanges one after another, on the rows they touch: the panel's
    // nb and the rows below it that some interchange brought in
    int own[kPanel], row[kPanel], from[kPanel], extra = 0;
    for (int c = 0; c < nb; ++c) own[c] = c;
    for (int c = 0; c < nb; ++c) {
      const int r = pivots[c];
      int* other;
      if (r < nb) {
        other = own + r;
      } else {
        int e = 0;
        while (e < extra && row[e] != r) ++e;
        if (e == extra) row[extra] = from[extra] = r, ++extra;
        other = from + e;
      }
      const int t = own[c];
      own[c] = *other;
      *other = t;
    }
    for (int c = 0; c < nb; ++c) perm->dst[c] = k0 + c, perm->src[c] = k0 + own[c];
    for (int e = 0; e < extra; ++e) perm->dst[nb + e] = k0 + row[e], perm->src[nb + e] = k0 + from[e];
    perm->count = nb + extra;
  }
}

// Sixteen lanes a column j outside the panel: the panel's interchanges, then,
// right of the panel, the panel's rows of U (unit lower triangle, k ascending).
template <class T>
__global__ void __launch_bounds__(128) k_lu_rows(T* A, int n, int k0, int nb,
                                                const Perm* perm) {
  after_previous();
  __shared__ T L[kPanel][kPanel + 1];
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) L[e % nb][e / nb] = A[(size_t)(k0 + e / nb) * n + k0 + e % nb];
  __syncthreads();
  const int lane = threadIdx.x & (kPanel - 1);
  int j = blockIdx.x * (128 / kPanel) + threadIdx.x / kPanel;
  const bool live = j < n - nb;
  if (j >= k0) j += nb;
  T* col = A + (size_t)(live ? j : 0) * n;
  const int count = perm->count;
  T v[2] = {(T)0, (T)0};
  for (int h = 0; h < 2; ++h)
    if (live && lane + h * kPanel < count) v[h] = col[perm->src[lane + h * kPanel]];
  __syncwarp();
  // entries 0 .. nb - 1 are the panel's rows; the solve takes them from lanes 0 .. nb - 1
  const bool right = j >= k0 + nb;
  T a = v[0];
  for (int k = 0; k < nb; ++k) {
    const T u = __shfl_sync(0xffffffffu, a, (threadIdx.x & 16) + k);
    if (right && lane > k && lane < nb) a = sub_mul(a, L[lane][k], u);
  }
  if (live) {
    if (lane < count) col[perm->dst[lane]] = a;
    if (lane + kPanel < count) col[perm->dst[lane + kPanel]] = v[1];
  }
}

// The trailing matrix, 32 x 16 elements a block, four a thread.
template <class T>
__global__ void __launch_bounds__(128) k_lu_update(T* A, int n, int k0, int nb) {
  after_previous();
  __shared__ T L[kPanel][32], U[kPanel][16];
  const int i0 = k0 + nb + blockIdx.x * 32, j0 = k0 + nb + blockIdx.y * 16;
  for (int e = threadIdx.x; e < nb * 32; e += 128)
    L[e >> 5][e & 31] = i0 + (e & 31) < n ? A[(size_t)(k0 + (e >> 5)) * n + i0 + (e & 31)] : (T)0;
  for (int e = threadIdx.x; e < nb * 16; e += 128)
    U[e % nb][e / nb] = j0 + e / nb < n ? A[(size_t)(j0 + e / nb) * n + k0 + e % nb] : (T)0;
  __syncthreads();
  const int i = threadIdx.x & 31, j = threadIdx.x >> 5;
  if (i0 + i >= n) return;
  T a[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = j0 + j + 4 * q < n ? A[(size_t)(j0 + j + 4 * q) * n + i0 + i] : (T)0;
  for (int k = 0; k < nb; ++k)
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = sub_mul(a[q], L[k][i], U[k][j + 4 * q]);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (j0 + j + 4 * q < n) A[(size_t)(j0 + j + 4 * q) * n + i0 + i] = a[q];
}

template <class T>
void lu(const double* AIC, T* A, int n, int* piv, int* err, Perm* perm, cudaStream_t st) {
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr[dev].load(std::memory_order_acquire)) {
    cudaFuncSetAttribute(k_lu_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (dev >= 0 && dev < 64) attr[dev].store(true, std::memory_order_release);
  }
  const size_t n2 = (size_t)n * n;
  count_launch();
  launch_next(k_lu_copy<T>, (unsigned)((n2 + 255) / 256), 256, 0, st, AIC, A, n2);
  for (int k0 = 0; k0 < n;) {
    // as many columns as fit shared memory (all kPanel up to 1800 rows)
    const int fit = (int)(kSmemMax / sizeof(T) / (size_t)(n - k0));
    const int nb = std::max(1, std::min(std::min(kPanel, fit), n - k0));
    count_launch();
    launch_next(k_lu_panel<T>, 1, kPanelThreads, sizeof(T) * nb * (size_t)(n - k0), st, A, n, k0, nb, piv, err, perm);
    if (n > nb) {
      count_launch();
      launch_next(k_lu_rows<T>, (n - nb + 128 / kPanel - 1) / (128 / kPanel), 128, 0, st, A, n, k0, nb, perm);
    }
    const int rest = n - k0 - nb;
    if (rest > 0) {
      count_launch();
      launch_next(k_lu_update<T>, dim3((rest + 31) / 32, (rest + 15) / 16), 128, 0, st, A, n, k0, nb);
    }
    k0 += nb;
  }
}

// ---- inverse ------------------------------------------------------------------
// X = A^-1 column by column (P e_c forward through L, then backward through U),
// kCols columns a block.  Forward, each column's sums run down the rows in
// parallel, k ascending.  Backward, X[i] = (X[i] - U[i][i+1] X[i+1] - U[i][i+2] X[i+2]
// - ...) / U[i][i] starts with the value found last, so its n^2 / 2 subtractions
// are one chain of 64 cycles each (1.4 ms at n = 300), which is all one warp does: the
// others have the products of the next row ready when the chain gets there.  The
// products and the rows of U were on the chain before: 9.1 ms.
constexpr int kInvThreads = 128;

__global__ void __launch_bounds__(kInvThreads) k_inverse64(const double* A, const int* piv,
                                                          int n, int cols, double* inv) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  double* X = reinterpret_cast<double*>(smem);  // [row][column]
  double* prod = X + (size_t)n * cols;          // [2][k][column]: products of a row's later columns
  double* U = prod + (size_t)2 * n * cols;      // [4][k]: rows of U on their way
  const int c0 = blockIdx.x * cols, nc = min(cols, n - c0);
  const int tid = threadIdx.x;
  for (int e = tid; e < n * cols; e += kInvThreads) X[e] = 0.0;
  __syncthreads();
  if (tid < nc) {
    int pos = c0 + tid;  // position of the 1 in P e_c after the row interchanges
    for (int k = 0; k < n; ++k) {
      const int pk = piv[k];
      if (pos == k) pos = pk;
      else if (pos == pk) pos = k;
    }
    X[(size_t)pos * cols + tid] = 1.0;
  }
  __syncthreads();
  // forward: the next column of L in registers while this one is used
  constexpr int kAhead = 4;
  double next[kAhead];
  auto fetch = [&](int k) {
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      const int i = k + 1 + tid + q * kInvThreads;
      next[q] = k < n && i < n ? A[(size_t)k * n + i] : 0.0;
    }
  };
  fetch(0);
  for (int k = 0; k < n; ++k) {
    double l[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) l[q] = next[q];
    fetch(k + 1);
    for (int c = 0; c < nc; ++c) {
      const double x = X[(size_t)k * cols + c];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int i = k + 1 + tid + q * kInvThreads;
        if (i < n) X[(size_t)i * cols + c] = sub_mul(X[(size_t)i * cols + c], l[q], x);
      }
      for (int i = k + 1 + tid + kAhead * kInvThreads; i < n; i += kInvThreads)
        X[(size_t)i * cols + c] = sub_mul(X[(size_t)i * cols + c], A[(size_t)k * n + i], x);
    }
    __syncthreads();
  }
  // backward
  auto load_row = [&](int i) {  // row i of U from the diagonal on
    if (i >= 0)
      for (int k = i + tid; k < n; k += kInvThreads) U[(size_t)(i & 3) * n + k] = A[(size_t)k * n + i];
  };
  load_row(n - 1);
  load_row(n - 2);
  load_row(n - 3);
  __syncthreads();
  for (int i = n - 1; i >= 0; --i) {
    if (tid < 32) {
      if (tid < nc) {
        const double* u = U + (size_t)(i & 3) * n;
        const double* p = prod + (size_t)(i & 1) * n * cols + tid;
        double s = X[(size_t)i * cols + tid];
        if (i + 1 < n) s = s - u[i + 1] * X[(size_t)(i + 1) * cols + tid];
#pragma unroll 8
        for (int k = i + 2; k < n; ++k) s = s - p[(size_t)k * cols];
        X[(size_t)i * cols + tid] = exact64::quotient(s, u[i]);
      }
    } else {
      // row i - 1's products with what is known: X[i + 1], X[i + 2], ...; row i - 3 of U
      if (i >= 1) {
        const double* u = U + (size_t)((i - 1) & 3) * n;
        double* p = prod + (size_t)((i - 1) & 1) * n * cols;
        for (int e = (i + 1) * cols + tid - 32; e < n * cols; e += kInvThreads - 32) p[e] = u[e / cols] * X[e];
      }
      if (i >= 3)
        for (int k = i - 3 + tid - 32; k < n; k += kInvThreads - 32)
          U[(size_t)((i - 3) & 3) * n + k] = A[(size_t)k * n + i - 3];
    }
    __syncthreads();
  }
  for (int e = tid; e < n * nc; e += kInvThreads) {
    const int c = e / n, i = e - c * n;
    inv[(size_t)(c0 + c) * n + i] = X[(size_t)i * cols + c];
  }
}

// The same, a thread per column on global memory: for matrices whose columns do
// not fit shared memory (over 4100 rows).  By time the line would lie lower, where
// a block is left with a column or two and the blocks come in waves: AIC, factors
// and inverse take 0.32 s at 1812 rows, 1.7 at 2800, 7.2 at 3700, and 3.4 this way
// at 4200 (with LU and inverse each in one launch 1.6, 5.4, 12.0 and 18.3 s).
__global__ void k_inverse64_big(const double* A, const int* piv, int n,
                                double* inv) {
  after_previous();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double* X = inv + (size_t)n * c;
  int pos = c;
  for (int k = 0; k < n; ++k) {
    const int pk = piv[k];
    if (pos == k) pos = pk;
    else if (pos == pk) pos = k;
  }
  for (int i = 0; i < n; ++i) {
    double sum = i == pos ? 1.0 : 0.0;
    for (int k = 0; k < i; ++k) sum = sum - A[i + (size_t)n * k] * X[k];
    X[i] = sum;
  }
  for (int i = n - 1; i >= 0; --i) {
    double sum = X[i];
    for (int k = i + 1; k < n; ++k) sum = sum - A[i + (size_t)n * k] * X[k];
    X[i] = sum / A[i + (size_t)n * i];
  }
}

// FP32: a warp per column, lanes over k.
__global__ void __launch_bounds__(128) k_inverse32(const float* A, const int* piv, int n,
                                                  float* inv) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int c = blockIdx.x * wpb + warp;
  if (c >= n) return;
  float* X = reinterpret_cast<float*>(smem) + (size_t)warp * n;
  int pos = c;
  for (int k = 0; k < n; ++k) {
    const int pk = piv[k];
    if (pos == k) pos = pk;
    else if (pos == pk) pos = k;
  }
  for (int i = 0; i < n; ++i) {
    float s = 0.f;
    for (int k = pos + lane; k < i; k += 32) s = fmaf(A[(size_t)k * n + i], X[k], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) X[i] = (i == pos ? 1.f : 0.f) - s;
    __syncwarp();
  }
  for (int i = n - 1; i >= 0; --i) {
    float s = 0.f;
    for (int k = i + 1 + lane; k < n; k += 32) s = fmaf(A[(size_t)k * n + i], X[k], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) X[i] = (X[i] - s) / A[(size_t)i * n + i];
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) inv[(size_t)c * n + i] = X[i];
}

// libMath.f90:428-458 (tolerance 1E-04 single precision)
__global__ void k_is_inverse(const double* A, const double* inv, int n, int* err) {
  after_previous();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)n * n) return;
  const int i = (int)(t % n), j = (int)(t / n);
  double sum = 0.0;
#pragma unroll 4
  for (int k = 0; k < n; ++k) sum = fma(A[i + (size_t)n * k], inv[k + (size_t)n * j], sum);
  const double tol = (double)1e-4f;
  const bool bad = (i != j) ? (sum > tol) : (sum - 1.0 > tol);
  if (bad) atomicExch(err, 11);
}

size_t inverse_smem(int n, int cols) { return sizeof(double) * ((size_t)3 * n * cols + (size_t)4 * n); }

}  // namespace

size_t lu_scratch_bytes() { return 2 * sizeof(Perm); }

void launch_lu_inverse(const Dims& d, const DevState& s, cudaStream_t st) {
  const int n = d.n;
  lu<double>(s.AIC, s.LU, n, s.piv, s.err, static_cast<Perm*>(s.luPerm), st);
  count_launch();
  if (inverse_smem(n, 1) > kSmemMax) {
    launch_next(k_inverse64_big, (n + 63) / 64, 64, 0, st, s.LU, s.piv, n, s.AICinv);
    return;
  }
  // as many columns a block as give every SM one, as far as shared memory holds them
  int cols = std::min(32, std::max(1, (n + device_sm_count() - 1) / device_sm_count()));
  while (cols > 1 && inverse_smem(n, cols) > kSmemMax) --cols;
  cudaFuncSetAttribute(k_inverse64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  launch_next(k_inverse64, (n + cols - 1) / cols, kInvThreads, inverse_smem(n, cols), st, s.LU, s.piv, n, cols, s.AICinv);
}

void launch_is_inverse(const Dims& d, const DevState& s, cudaStream_t st) {
  const long n2 = (long)d.n * d.n;
  count_launch();
  launch_next(k_is_inverse, (unsigned)((n2 + 255) / 256), 256, 0, st, s.AIC, s.AICinv, d.n, s.err);
}

void launch_lu32(const Dims& d, const DevState& s, cudaStream_t st) {
  const int n = d.n;
  lu<float>(s.AIC, s.LU32, n, s.piv32, nullptr, static_cast<Perm*>(s.luPerm) + 1, st);
  int wpb = 4;
  while (wpb > 1 && sizeof(float) * wpb * (size_t)n > 48 * 1024) --wpb;
  count_launch();
  launch_next(k_inverse32, (n + wpb - 1) / wpb, 32 * wpb, sizeof(float) * wpb * (size_t)n, st, s.LU32, s.piv32, n,
              s.AICinv32);
}

}  // namespace vlm
