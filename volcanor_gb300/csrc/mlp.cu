// MLP engine of the learned far-wake surrogate (see mlp.h): FP32 CUDA-core
// kernels for forward, backward and Adam, and the vlm_mlp_* C ABI.
//
// GEMM: C[M x N] = op(A)[M x K] op(B)[K x N] (+ bias, + tanh; or times the
// tanh derivative), 128 x 64 output tile per 256-thread block, 8 x 4 outputs per
// thread (three 16-byte shared loads per 32 FMAs; 4 x 4 needed four), K in steps
// of 16 through two shared buffers, the next step's global loads in flight behind
// the FMAs.  Each output sums k = 0..K-1 in order, so results do not depend on
// the launch configuration.
//
// The weight gradients are GEMMs over the batch (K = thousands of rows, M x N =
// one or two tiles): one block each took 5.3 ms at 20000 rows.  They run in
// slices of the batch, one block per tile and slice, whose sums (and the bias
// gradients', summed from the same staged rows) one kernel adds in slice order.
// The slices depend on the batch size and the network alone, so training is
// reproducible.  20000 rows of a 12-128-128-128-3 network from host arrays:
// 12.8 -> 0.40 ms, gradient error against 64 bits 2.1e-6 -> 4.3e-7.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/vlm.h"
#include "mlp.h"
#include "vlm_bs.h"

namespace vlm {

extern thread_local std::string g_err;

namespace {

#define MLP_CUDA(x)                                                                        \
  do {                                                                                     \
    cudaError_t e_ = (x);                                                                  \
    if (e_ != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + cudaGetErrorString(e_)); \
  } while (0)

enum { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_TANH = 2, EPI_TANH_BACK = 3 };
constexpr int kBM = 128, kBN = 64, kBK = 16;

// bias: the row vector added (EPI_BIAS*); H: activations whose tanh derivative
// 1 - H^2 multiplies the result (EPI_TANH_BACK, laid out as C).  SLICES: the
// block sums rows kslice blockIdx.z .. of the K dimension only, into its own copy
// of C (cstride floats apart), and with rowsum the column sums of A as well.
template <bool TA, bool TB, int EPI, bool SLICES>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, const float* __restrict__ A, int lda,
                                              const float* __restrict__ B, int ldb, float* __restrict__ C, int ldc,
                                              const float* __restrict__ bias, const float* __restrict__ H, int kslice,
                                              int64_t cstride, float* __restrict__ rowsum) {
  __shared__ __align__(16) float As[2][kBK][kBM + 4];
  __shared__ __align__(16) float Bs[2][kBK][kBN + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  const int kb = SLICES ? (int)blockIdx.z * kslice : 0, ke = SLICES ? min(K, kb + kslice) : K;
  float acc[8][4], rs[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    rs[i] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  }
  float ra[8], rb[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = threadIdx.x + 256 * q;
      const int mm = TA ? e & (kBM - 1) : e >> 4, kk = TA ? e >> 7 : e & 15;
      const int gm = m0 + mm, gk = k0 + kk;
      ra[q] = gm < M && gk < ke ? (TA ? A[(size_t)gk * lda + gm] : A[(size_t)gm * lda + gk]) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = threadIdx.x + 256 * q;
      const int nn = TB ? e >> 4 : e & (kBN - 1), kk = TB ? e & 15 : e >> 6;
      const int gn = n0 + nn, gk = k0 + kk;
      rb[q] = gn < N && gk < ke ? (TB ? B[(size_t)gn * ldb + gk] : B[(size_t)gk * ldb + gn]) : 0.f;
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = threadIdx.x + 256 * q;
      As[buf][TA ? e >> 7 : e & 15][TA ? e & (kBM - 1) : e >> 4] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = threadIdx.x + 256 * q;
      Bs[buf][TB ? e & 15 : e >> 6][TB ? e >> 4 : e & (kBN - 1)] = rb[q];
    }
  };
  fetch(kb);
  stage(0);
  __syncthreads();
  for (int k0 = kb, buf = 0; k0 < ke; k0 += kBK, buf ^= 1) {
    const bool more = k0 + kBK < ke;
    if (more) fetch(k0 + kBK);
#pragma unroll
    for (int kk = 0; kk < kBK; ++kk) {
      float a[8], b[4];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8]);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8 + 4]);
      *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (SLICES) rs[i] += a[i];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
    }
    if (more) stage(buf ^ 1);
    __syncthreads();
  }
  if (SLICES) C += (int64_t)blockIdx.z * cstride;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gm = m0 + ty * 8 + i;
    if (gm >= M) continue;
    if (SLICES && n0 == 0 && tx == 0) rowsum[(int64_t)blockIdx.z * cstride + gm] = rs[i];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float c = acc[i][j];
      if (EPI == EPI_BIAS || EPI == EPI_BIAS_TANH) c += bias[gn];
      if (EPI == EPI_BIAS_TANH) c = tanhf(c);
      if (EPI == EPI_TANH_BACK) {
        const float h = H[(size_t)gm * ldc + gn];
        c = c * (1.f - h * h);
      }
      C[(size_t)gm * ldc + gn] = c;
    }
  }
}

template <bool TA, bool TB, int EPI>
void gemm(cudaStream_t st, int M, int N, int K, const float* A, int lda, const float* B, int ldb, float* C, int ldc,
          const float* bias, const float* H = nullptr) {
  if (M <= 0 || N <= 0) return;
  dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM);
  count_launch();
  k_gemm<TA, TB, EPI, false><<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, H, 0, 0, nullptr);
}

// Rows of the batch a slice of the weight gradients sums: 128 (enough slices to
// fill the device from about 10000 rows on), more when that made over 64 slices
// or over 2^26 partial sums (a wide network's tiles fill the device by themselves).
int slice_rows(int n, int64_t nparam) {
  const int most = (int)std::max<int64_t>(1, std::min<int64_t>(64, ((int64_t)1 << 26) / nparam));
  const int r = std::max(128, (n + most - 1) / most);
  return (r + kBK - 1) / kBK * kBK;
}

// g[i] = the slices' sums added in slice order
__global__ void k_sum_slices(const float* __restrict__ part, int64_t stride, int slices, int64_t n,
                             float* __restrict__ g) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = part[i];
#pragma unroll 8
  for (int k = 1; k < slices; ++k) s += part[(int64_t)k * stride + i];
  g[i] = s;
}

// dY = 2 (Y - T) / (rows x cols); per-block partial sums of (Y - T)^2
constexpr int kLossThreads = 256;
__global__ void k_mse(const float* __restrict__ Y, const float* __restrict__ T, int64_t n, float scale,
                      float* __restrict__ dY, float* __restrict__ part) {
  __shared__ float red[kLossThreads];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  float e2 = 0.f;
  if (i < n) {
    const float e = Y[i] - T[i];
    dY[i] = 2.f * e * scale;
    e2 = e * e;
  }
  red[threadIdx.x] = e2;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}
__global__ void k_sum_parts(const float* __restrict__ part, int n, float scale, float* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  float s = 0.f;
  for (int i = 0; i < n; ++i) s += part[i];
  out[0] = s * scale;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

void MlpShape::finalize() {
  nparam = 0;
  maxw = 0;
  for (int l = 0; l < nl; ++l) {
    woff[l] = nparam;
    nparam += (int64_t)sz[l + 1] * sz[l];
    boff[l] = nparam;
    nparam += sz[l + 1];
  }
  for (int l = 0; l <= nl; ++l) maxw = std::max(maxw, sz[l]);
}

void Mlp::create(const std::vector<int>& sizes, uint64_t seed, cudaStream_t stream) {
  if (sizes.size() < 2 || (int)sizes.size() > kMlpMaxLayers + 1) throw std::invalid_argument("MLP needs 2..9 layer sizes");
  for (int s : sizes)
    if (s <= 0 || s > 4096) throw std::invalid_argument("MLP layer sizes must be in [1, 4096]");
  st = stream;
  sh.nl = (int)sizes.size() - 1;
  for (size_t i = 0; i < sizes.size(); ++i) sh.sz[i] = sizes[i];
  sh.finalize();
  // Glorot-uniform weights from a seeded generator, zero biases
  std::vector<float> h((size_t)sh.nparam, 0.f);
  uint64_t s = seed;
  for (int l = 0; l < sh.nl; ++l) {
    const double a = std::sqrt(6.0 / (sh.sz[l] + sh.sz[l + 1]));
    for (int64_t i = 0; i < (int64_t)sh.sz[l + 1] * sh.sz[l]; ++i) {
      const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
      h[(size_t)(sh.woff[l] + i)] = (float)((2.0 * u - 1.0) * a);
    }
  }
  MLP_CUDA(cudaMalloc(&p, sizeof(float) * sh.nparam));
  MLP_CUDA(cudaMalloc(&g, sizeof(float) * sh.nparam));
  MLP_CUDA(cudaMalloc(&m, sizeof(float) * sh.nparam));
  MLP_CUDA(cudaMalloc(&v, sizeof(float) * sh.nparam));
  MLP_CUDA(cudaMalloc(&loss, sizeof(float) * 2));
  // on the network's own stream: a case's does not wait for the legacy one
  MLP_CUDA(cudaMemcpyAsync(p, h.data(), sizeof(float) * sh.nparam, cudaMemcpyHostToDevice, st));
  MLP_CUDA(cudaMemsetAsync(g, 0, sizeof(float) * sh.nparam, st));
  MLP_CUDA(cudaMemsetAsync(m, 0, sizeof(float) * sh.nparam, st));
  MLP_CUDA(cudaMemsetAsync(v, 0, sizeof(float) * sh.nparam, st));
  adamStep = 0;
  tcFits = tc.plan(sh);
  if (tcFits) {
    MLP_CUDA(cudaMalloc(&tcImg, tc.imgBytes));
    MLP_CUDA(cudaMalloc(&tcErr, sizeof(int)));
    MLP_CUDA(cudaMemsetAsync(tcErr, 0, sizeof(int), st));
  }
  useTc = tcFits;
  tcStale = true;
}

bool Mlp::setTensorCores(bool on) {
  if (on && !tcFits) return false;
  useTc = on;
  return true;
}

void Mlp::destroy() {
  for (float* q : {p, g, m, v, act, dact, loss, part, gpart})
    if (q) cudaFree(q);
  p = g = m = v = act = dact = loss = part = gpart = nullptr;
  gslices = 0;
  if (tcImg) cudaFree(tcImg);
  if (tcErr) cudaFree(tcErr);
  tcImg = nullptr;
  tcErr = nullptr;
  cap = 0;
}

void Mlp::reserve(int batch) {
  if (batch <= cap) return;
  if (act) cudaFree(act);
  if (dact) cudaFree(dact);
  if (part) cudaFree(part);
  act = dact = part = nullptr;
  MLP_CUDA(cudaMalloc(&act, sizeof(float) * (size_t)(sh.nl + 1) * batch * sh.maxw));
  MLP_CUDA(cudaMalloc(&dact, sizeof(float) * (size_t)2 * batch * sh.maxw));
  MLP_CUDA(cudaMalloc(&part, sizeof(float) * (size_t)((int64_t)batch * sh.maxw / kLossThreads + 2)));
  cap = batch;
}

void Mlp::forward(const float* X, int n, float* Y) {
  if (useTc) {
    if (tcStale) {
      tc_pack(p, sh, tc, tcImg, st);
      tcStale = false;
    }
    tc_forward(tc, tcImg, X, n, Y, tcErr, st);
    return;
  }
  const int chunk = std::max(cap, 1);
  for (int r0 = 0; r0 < n; r0 += chunk) {
    const int rows = std::min(chunk, n - r0);
    const float* H = X + (size_t)r0 * sh.sz[0];
    for (int l = 0; l < sh.nl; ++l) {
      const int in = sh.sz[l], out = sh.sz[l + 1];
      const bool last = l == sh.nl - 1;
      float* Z = last ? Y + (size_t)r0 * out : act + (size_t)(l + 1) * cap * sh.maxw;
      if (last) gemm<false, true, EPI_BIAS>(st, rows, out, in, H, in, p + sh.woff[l], in, Z, out, p + sh.boff[l]);
      else gemm<false, true, EPI_BIAS_TANH>(st, rows, out, in, H, in, p + sh.woff[l], in, Z, out, p + sh.boff[l]);
      H = Z;
    }
  }
}

void Mlp::grad(const float* X, const float* T, int n) {
  reserve(n);
  // forward, keeping every layer's output (layer 0 = X)
  const float* Hs[kMlpMaxLayers + 1];
  Hs[0] = X;
  for (int l = 0; l < sh.nl; ++l) {
    const int in = sh.sz[l], out = sh.sz[l + 1];
    float* Z = act + (size_t)(l + 1) * cap * sh.maxw;
    if (l == sh.nl - 1) gemm<false, true, EPI_BIAS>(st, n, out, in, Hs[l], in, p + sh.woff[l], in, Z, out, p + sh.boff[l]);
    else gemm<false, true, EPI_BIAS_TANH>(st, n, out, in, Hs[l], in, p + sh.woff[l], in, Z, out, p + sh.boff[l]);
    Hs[l + 1] = Z;
  }
  // loss and dY
  const int out = sh.sz[sh.nl];
  const int64_t ny = (int64_t)n * out;
  float* dZ = dact;
  const int nb = (int)((ny + kLossThreads - 1) / kLossThreads);
  count_launch();
  k_mse<<<nb, kLossThreads, 0, st>>>(Hs[sh.nl], T, ny, 1.f / (float)ny, dZ, part);
  count_launch();
  k_sum_parts<<<1, 32, 0, st>>>(part, nb, 1.f / (float)ny, loss);
  // backward
  const int rows = slice_rows(n, sh.nparam), slices = (n + rows - 1) / rows;
  if (slices > gslices) {
    if (gpart) MLP_CUDA(cudaFree(gpart));
    gpart = nullptr;
    gslices = 0;
    MLP_CUDA(cudaMalloc(&gpart, sizeof(float) * (size_t)sh.nparam * slices));
    gslices = slices;
  }
  for (int l = sh.nl - 1; l >= 0; --l) {
    const int in = sh.sz[l], o = sh.sz[l + 1];
    // dW = dZ^T H_prev and db = column sums of dZ, in slices of the batch
    dim3 grid((in + kBN - 1) / kBN, (o + kBM - 1) / kBM, slices);
    count_launch();
    k_gemm<true, false, EPI_NONE, true><<<grid, 256, 0, st>>>(o, in, n, dZ, o, Hs[l], in, gpart + sh.woff[l], in,
                                                             nullptr, nullptr, rows, sh.nparam, gpart + sh.boff[l]);
    if (l > 0) {
      float* dH = (dZ == dact) ? dact + (size_t)cap * sh.maxw : dact;
      // through the weights and the layer below's tanh
      gemm<false, false, EPI_TANH_BACK>(st, n, in, o, dZ, o, p + sh.woff[l], in, dH, in, nullptr, Hs[l]);
      dZ = dH;
    }
  }
  count_launch();
  k_sum_slices<<<(unsigned)((sh.nparam + 255) / 256), 256, 0, st>>>(gpart, sh.nparam, slices, sh.nparam, g);
}

void Mlp::adam(float lr, float b1, float b2, float eps) {
  ++adamStep;
  tcStale = true;
  const float c1 = 1.f - std::pow(b1, (float)adamStep), c2 = 1.f - std::pow(b2, (float)adamStep);
  count_launch();
  k_adam<<<(unsigned)((sh.nparam + 255) / 256), 256, 0, st>>>(p, g, m, v, sh.nparam, lr, b1, b2, eps, c1, c2);
}

}  // namespace vlm

// ---------------------------------------------------------------------------
// C ABI (no counterpart in the reference: the learned part of this engine)
using namespace vlm;

struct vlm_mlp {
  Mlp net;
  float* dX = nullptr;
  float* dT = nullptr;
  float* dY = nullptr;
  int64_t capX = 0, capT = 0, capY = 0;
  ~vlm_mlp() {
    net.destroy();
    for (float* q : {dX, dT, dY})
      if (q) cudaFree(q);
  }
};

template <class F>
static int mlp_guard(F f) {
  try {
    f();
    return VLM_OK;
  } catch (const std::invalid_argument& e) {
    g_err = e.what();
    return VLM_ERR_INVALID;
  } catch (const std::exception& e) {
    g_err = e.what();
    return VLM_ERR_CUDA;
  }
}

static void grow_dev(float** q, int64_t& cap, int64_t n) {
  if (n <= cap) return;
  if (*q) cudaFree(*q);
  *q = nullptr;
  MLP_CUDA(cudaMalloc(q, sizeof(float) * (size_t)n));
  cap = n;
}

extern "C" int vlm_mlp_create(const int* sizes, int nsizes, uint64_t seed, vlm_mlp** out) {
  if (!sizes || !out || nsizes < 2) return VLM_ERR_INVALID;
  return mlp_guard([&]() {
    vlm_mlp* h = new vlm_mlp();
    try {
      h->net.create(std::vector<int>(sizes, sizes + nsizes), seed, nullptr);
    } catch (...) {
      delete h;
      throw;
    }
    *out = h;
  });
}

extern "C" int vlm_mlp_destroy(vlm_mlp* h) {
  delete h;
  return VLM_OK;
}

extern "C" int64_t vlm_mlp_param_count(const vlm_mlp* h) { return h ? h->net.sh.nparam : -1; }

extern "C" int vlm_mlp_get_params(vlm_mlp* h, float* out) {
  if (!h || !out) return VLM_ERR_INVALID;
  return mlp_guard([&]() {
    MLP_CUDA(cudaMemcpy(out, h->net.p, sizeof(float) * h->net.sh.nparam, cudaMemcpyDeviceToHost));
  });
}

extern "C" int vlm_mlp_set_params(vlm_mlp* h, const float* in) {
  if (!h || !in) return VLM_ERR_INVALID;
  return mlp_guard([&]() {
    MLP_CUDA(cudaMemcpy(h->net.p, in, sizeof(float) * h->net.sh.nparam, cudaMemcpyHostToDevice));
    h->net.tcStale = true;
  });
}

extern "C" int vlm_mlp_set_inference(vlm_mlp* h, int mode) {
  if (!h || mode < 0 || mode > 1) return VLM_ERR_INVALID;
  if (!h->net.setTensorCores(mode == 1)) {
    g_err = "vlm_mlp_set_inference: the network does not fit the tensor-core kernel (a layer wider than 256)";
    return VLM_ERR_UNSUPPORTED;
  }
  return VLM_OK;
}

extern "C" int vlm_mlp_get_inference(const vlm_mlp* h) { return h ? (h->net.useTc ? 1 : 0) : -1; }

extern "C" int vlm_mlp_forward(vlm_mlp* h, const float* X, int64_t n, float* Y) {
  if (!h || n < 0 || (n > 0 && (!X || !Y)) || n > (1 << 28)) return VLM_ERR_INVALID;
  if (n == 0) return VLM_OK;
  return mlp_guard([&]() {
    const int in = h->net.sh.sz[0], out = h->net.sh.sz[h->net.sh.nl];
    grow_dev(&h->dX, h->capX, n * in);
    grow_dev(&h->dY, h->capY, n * out);
    h->net.reserve((int)std::min<int64_t>(n, 1 << 16));
    MLP_CUDA(cudaMemcpy(h->dX, X, sizeof(float) * n * in, cudaMemcpyHostToDevice));
    h->net.forward(h->dX, (int)n, h->dY);
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpy(Y, h->dY, sizeof(float) * n * out, cudaMemcpyDeviceToHost));
    if (h->net.useTc) {
      int e = 0;
      MLP_CUDA(cudaMemcpy(&e, h->net.tcErr, sizeof(int), cudaMemcpyDeviceToHost));
      if (e) {
        MLP_CUDA(cudaMemset(h->net.tcErr, 0, sizeof(int)));
        throw std::runtime_error("tensor-core MLP: a bounded wait expired");
      }
    }
  });
}

extern "C" int vlm_mlp_gradient(vlm_mlp* h, const float* X, const float* T, int64_t n, float* grad, float* loss) {
  if (!h || !X || !T || !grad || n <= 0 || n > (1 << 22)) return VLM_ERR_INVALID;
  return mlp_guard([&]() {
    const int in = h->net.sh.sz[0], out = h->net.sh.sz[h->net.sh.nl];
    grow_dev(&h->dX, h->capX, n * in);
    grow_dev(&h->dT, h->capT, n * out);
    MLP_CUDA(cudaMemcpy(h->dX, X, sizeof(float) * n * in, cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemcpy(h->dT, T, sizeof(float) * n * out, cudaMemcpyHostToDevice));
    h->net.grad(h->dX, h->dT, (int)n);
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpy(grad, h->net.g, sizeof(float) * h->net.sh.nparam, cudaMemcpyDeviceToHost));
    if (loss) MLP_CUDA(cudaMemcpy(loss, h->net.loss, sizeof(float), cudaMemcpyDeviceToHost));
  });
}

extern "C" int vlm_mlp_train(vlm_mlp* h, const float* X, const float* T, int64_t n, int batch, int iters, float lr,
                             float* final_loss) {
  if (!h || !X || !T || n <= 0 || batch <= 0 || iters < 0 || n > (1 << 26)) return VLM_ERR_INVALID;
  return mlp_guard([&]() {
    const int in = h->net.sh.sz[0], out = h->net.sh.sz[h->net.sh.nl];
    grow_dev(&h->dX, h->capX, n * in);
    grow_dev(&h->dT, h->capT, n * out);
    MLP_CUDA(cudaMemcpy(h->dX, X, sizeof(float) * n * in, cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemcpy(h->dT, T, sizeof(float) * n * out, cudaMemcpyHostToDevice));
    const int b = (int)std::min<int64_t>(batch, n);
    const int64_t nbatch = n / b;
    for (int it = 0; it < iters; ++it) {
      const int64_t k = it % std::max<int64_t>(nbatch, 1);  // consecutive batches of the (pre-shuffled) set
      h->net.grad(h->dX + (size_t)k * b * in, h->dT + (size_t)k * b * out, b);
      h->net.adam(lr);
    }
    MLP_CUDA(cudaGetLastError());
    if (final_loss) {
      MLP_CUDA(cudaStreamSynchronize(h->net.st));
      MLP_CUDA(cudaMemcpy(final_loss, h->net.loss, sizeof(float), cudaMemcpyDeviceToHost));
    }
  });
}
