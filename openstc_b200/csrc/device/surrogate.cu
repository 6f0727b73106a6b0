// Chemistry surrogate: data generation with the FP64 EPI step, training with
// the tcgen05 layer kernels of mlp_train.cuh, the plain BF16 GEMM, and the host
// side of the fused tensor-core inference behind a trust gate.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <limits>
#include <algorithm>
#include <random>
#include <stdexcept>
#include <string>

#include "engine.hpp"
#include "kernels_surrogate.cuh"
#include "mlp_train.cuh"
#include "openstc_b200.h"
#include "surrogate.hpp"
#include "tc_gemm.cuh"

namespace ostc {

// Device-to-host copy ordered after the work on stream_ (a plain cudaMemcpy
// runs on the legacy default stream, which does not wait for this
// non-blocking stream).
#define d2h(dst, src, bytes, what)                                                              \
  do {                                                                                          \
    ck(cudaMemcpyAsync((dst), (src), (bytes), cudaMemcpyDeviceToHost, stream_), what);          \
    ck(cudaStreamSynchronize(stream_), what);                                                   \
  } while (0)

// ------------------------------------------------------------------ GEMM
template <int BN>
static cudaError_t launch_gemm_bn(const uint16_t *A, int lda, const uint16_t *B, int ldb, float *D, int ldd, int M,
                                  int N, int K, int splits, int *err, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_tc_gemm<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(GemmTile<BN>::smem));
  if (e != cudaSuccess) return e;
  const int per = (K + splits - 1) / splits;
  const int kps = (per + kGemmBK - 1) / kGemmBK * kGemmBK;
  const dim3 grid((M + 127) / 128, (N + BN - 1) / BN, splits);
  k_tc_gemm<BN><<<grid, 128, GemmTile<BN>::smem, st>>>(A, lda, B, ldb, D, ldd, M, N, K, kps, err);
  return cudaGetLastError();
}

// D = A * B^T on the tensor cores; with splits > 1, D holds `splits`
// consecutive partial results of M x ldd each.
cudaError_t tc_gemm(const uint16_t *A, int lda, const uint16_t *B, int ldb, float *D, int ldd, int M, int N, int K,
                    int splits, int *err, cudaStream_t st) {
  if (N <= 16) return launch_gemm_bn<16>(A, lda, B, ldb, D, ldd, M, N, K, splits, err, st);
  if (N <= 32) return launch_gemm_bn<32>(A, lda, B, ldb, D, ldd, M, N, K, splits, err, st);
  if (N <= 64) return launch_gemm_bn<64>(A, lda, B, ldb, D, ldd, M, N, K, splits, err, st);
  if (N <= 128) return launch_gemm_bn<128>(A, lda, B, ldb, D, ldd, M, N, K, splits, err, st);
  return launch_gemm_bn<256>(A, lda, B, ldb, D, ldd, M, N, K, splits, err, st);
}

namespace {

using Chem = Cfg<2, 1, 9>;
constexpr int NS = 9;

void ck(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}

// A temporary device array, freed when it leaves scope (an exception from a
// failed check included; cudaFree waits for the work still using it).
template <class T>
struct DevTemp {
  T *p = nullptr;
  DevTemp(size_t count, const char *what) { ck(cudaMalloc(&p, count * sizeof(T)), what); }
  ~DevTemp() { cudaFree(p); }
  DevTemp(const DevTemp &) = delete;
  DevTemp &operator=(const DevTemp &) = delete;
};

__host__ __device__ inline uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__device__ inline double u01(uint64_t &s) {
  s = mix64(s);
  return (static_cast<double>(s >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}
__device__ inline double gauss(uint64_t &s) {
  const double a = u01(s), b = u01(s);
  return sqrt(-2.0 * log(a)) * cos(6.283185307179586 * b);
}

__device__ inline uint16_t bf16(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }

// ------------------------------------------------------------------ samples
// T, p, Y[9], dt per sample: from the cells of a flow field (perturbed) or
// uniform in the training box with Dirichlet(1) mass fractions.
__global__ void k_sample(double *states, int64_t n, uint64_t seed, DevBlock F, int use_field, double field_fraction,
                         SurrogateGate g) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  uint64_t s = mix64(seed ^ mix64(static_cast<uint64_t>(i) + 1));
  double T, p, Y[NS];
  double dt = pow(10.0, g.ldt_min + (g.ldt_max - g.ldt_min) * u01(s));
  if (use_field && u01(s) < field_fraction) {
    const int64_t cells = static_cast<int64_t>(F.mx) * F.my * F.mz;
    int64_t c = static_cast<int64_t>(u01(s) * cells);
    if (c >= cells) c = cells - 1;
    const int ci = static_cast<int>(c % F.mx), cj = static_cast<int>((c / F.mx) % F.my),
              ck = static_cast<int>(c / (static_cast<int64_t>(F.mx) * F.my));
    const int64_t m = F.G.at(ci, cj, ck), sz = F.G.size;
    T = F.bv[5 * sz + m] * (1.0 + 0.02 * gauss(s));
    p = F.bv[4 * sz + m] * (1.0 + 0.02 * gauss(s));
    double sum = 0;
    for (int k = 0; k < NS; ++k) {
      Y[k] = fmax(F.sv[k * sz + m], 0.0) * exp(0.1 * gauss(s));
      sum += Y[k];
    }
    for (int k = 0; k < NS; ++k) Y[k] /= sum;
    // the cell's own local time step, perturbed within a factor of 2
    const double dtc = F.dt_local[F.Z.at(ci, cj, ck)];
    if (dtc > 0) dt = dtc * pow(10.0, 0.6 * u01(s) - 0.3);
  } else {
    T = g.t_min + (g.t_max - g.t_min) * u01(s);
    p = pow(10.0, g.lp_min + (g.lp_max - g.lp_min) * u01(s));
    double sum = 0;
    for (int k = 0; k < NS; ++k) {
      Y[k] = -log(u01(s));
      sum += Y[k];
    }
    for (int k = 0; k < NS; ++k) Y[k] /= sum;
  }
  T = fmin(fmax(T, static_cast<double>(g.t_min)), static_cast<double>(g.t_max));
  p = fmin(fmax(p, pow(10.0, static_cast<double>(g.lp_min))), pow(10.0, static_cast<double>(g.lp_max)));
  double *o = states + i * kSurIn;
  o[0] = T;
  o[1] = p;
  for (int k = 0; k < NS; ++k) o[2 + k] = Y[k];
  o[11] = dt;
}

template <class M>
__global__ void __launch_bounds__(128) k_label(const double *states, double *dy, int64_t n) {
  extern __shared__ double sq[];
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const double *s = states + i * kSurIn;
  double Y[NS], d[NS], mw_inv = 0;
  for (int k = 0; k < NS; ++k) {
    Y[k] = s[2 + k];
    mw_inv += div_mw(Y[k], k);
  }
  const double rho = s[1] / (kDR_u * s[0] * mw_inv);
  sur::epi_increment<NS, M>(s[0], rho, Y, s[11], sq + threadIdx.x, sq + cP.nr * blockDim.x + threadIdx.x, blockDim.x, d);
  for (int k = 0; k < NS; ++k) dy[i * NS + k] = d[k];
}

// ------------------------------------------------------------ normalisation
__device__ inline void raw_features(const double *s, float *f) {
  f[0] = static_cast<float>(s[0]);
  f[1] = static_cast<float>(log10(s[1]));
  for (int k = 0; k < NS; ++k) f[2 + k] = static_cast<float>(s[2 + k]);
  f[11] = static_cast<float>(log10(s[11]));
}

// sums of features, squared features and squared labels (double atomics)
__global__ void k_stats(const double *states, const double *dy, int64_t n, double *acc) {
  __shared__ double sh[2 * kSurIn + kSurOut];
  for (int q = threadIdx.x; q < 2 * kSurIn + kSurOut; q += blockDim.x) sh[q] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f[kSurIn];
    raw_features(states + i * kSurIn, f);
    for (int q = 0; q < kSurIn; ++q) {
      atomicAdd(&sh[q], static_cast<double>(f[q]));
      atomicAdd(&sh[kSurIn + q], static_cast<double>(f[q]) * f[q]);
    }
    for (int q = 0; q < kSurOut; ++q) atomicAdd(&sh[2 * kSurIn + q], dy[i * NS + q] * dy[i * NS + q]);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < 2 * kSurIn + kSurOut; q += blockDim.x) atomicAdd(&acc[q], sh[q]);
}

// features x = (f - mu) / sig; targets t_k = asinh(r_k / c_k) / s_k of the
// relative increments r_k = dY_k / (Y_k + eps) (the signed-log transform tames
// their heavy tail)
struct Norm {
  float mu[kSurIn], sig[kSurIn], c[kSurOut], s[kSurOut];
};

__global__ void k_features(const double *states, const double *dy, int64_t n, Norm nm, uint16_t *x, float *t) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  float f[kSurIn];
  raw_features(states + i * kSurIn, f);
  for (int q = 0; q < kSurInPad; ++q) x[i * kSurInPad + q] = q < kSurIn ? bf16((f[q] - nm.mu[q]) / nm.sig[q]) : 0;
  if (t)
    for (int q = 0; q < kSurOutPad; ++q)
      t[i * kSurOutPad + q] =
          q < kSurOut ? static_cast<float>(asinh(dy[i * NS + q] / (states[i * kSurIn + 2 + q] + kSurYEps) / nm.c[q]) / nm.s[q])
                      : 0.f;
}

// ---------------------------------------------------------------- training
// Rows of the batch into the first layer's operand image and the target
// buffer: row i of the data (in order; rows past n are zero) or a random one
// of its n rows.
__global__ void k_gather(const uint16_t *x, const float *t, int64_t n, uint64_t seed, bool in_order, int batch,
                         uint8_t *a0, float *tb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= batch) return;
  const int64_t src = in_order ? i : static_cast<int64_t>(mix64(seed ^ mix64(static_cast<uint64_t>(i) + 7)) % n);
  const bool live = src < n;
  const uint4 *xs = reinterpret_cast<const uint4 *>(x + src * kSurInPad);
  uint8_t *img = a0 + static_cast<int64_t>(i / mlp::kTile) * mlp::kChunk;
  for (int p = 0; p < 2; ++p)
    *reinterpret_cast<uint4 *>(img + mlp::image_offset(mlp::kTile, i % mlp::kTile, 8 * p)) =
        live ? xs[p] : make_uint4(0, 0, 0, 0);
  if (!t) return;
  const float4 *ts = reinterpret_cast<const float4 *>(t + src * kSurOutPad);
  float4 *to = reinterpret_cast<float4 *>(tb + static_cast<int64_t>(i) * kSurOutPad);
  for (int p = 0; p < kSurOutPad / 4; ++p) to[p] = live ? ts[p] : make_float4(0, 0, 0, 0);
}

// bf16 copies of a weight [dout x din]: the operand image of the training
// kernels and the tile order of the fused inference kernel (K chunks of 16
// columns).
__global__ void k_pack(const float *w, int dout, int din, uint8_t *img, uint8_t *wp) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<int64_t>(dout) * din) return;
  const int r = static_cast<int>(i / din), k = static_cast<int>(i % din);
  const uint16_t v = bf16(w[i]);
  *reinterpret_cast<uint16_t *>(img + mlp::image_offset(dout, r, k)) = v;
  const int bk = 16;
  const int c = k / bk, kk = k % bk;
  *reinterpret_cast<uint16_t *>(wp + static_cast<size_t>(c) * dout * bk * 2 + tc::tile_offset(r, kk, bk)) = v;
}

}  // namespace

// ================================================================ Surrogate
Surrogate::Surrogate(const DevParams &chem, const std::vector<int> &elem_comp, int n_elem, int device, uint64_t seed)
    : chem_(chem), elem_comp_(elem_comp), n_elem_(n_elem), device_(device), seed_(seed) {
  if (chem.ns != NS || chem.mix != 2) throw std::runtime_error("the surrogate is built for the 9-species finite-rate mechanism");
  if (n_elem > kMaxElem) throw std::runtime_error("too many elements for the surrogate's conservation gate");
  ck(cudaSetDevice(device), "cudaSetDevice");
  ck(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "stream");
  const int dims[kSurLayers + 1] = {kSurInPad, kSurHidden, kSurHidden, kSurHidden, kSurHidden, kSurOutPad};
  std::mt19937_64 rng(seed);
  for (int l = 0; l < kSurLayers; ++l) {
    din_[l] = dims[l];
    dout_[l] = dims[l + 1];
    const size_t nw = static_cast<size_t>(dout_[l]) * din_[l];
    const int fan_in = l == 0 ? kSurIn : din_[l];
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / fan_in) * (l == kSurLayers - 1 ? 0.5f : 1.f));
    std::vector<float> w(nw, 0.f), b(dout_[l], 0.f);
    const int valid_out = l == kSurLayers - 1 ? kSurOut : dout_[l];
    for (int r = 0; r < valid_out; ++r)
      for (int k = 0; k < fan_in; ++k) w[static_cast<size_t>(r) * din_[l] + k] = nd(rng);
    auto alloc = [&](size_t bytes) {
      void *p = nullptr;
      ck(cudaMalloc(&p, bytes), "cudaMalloc surrogate");
      ck(cudaMemsetAsync(p, 0, bytes, stream_), "memset surrogate");
      allocs_.push_back(p);
      return p;
    };
    w_[l] = static_cast<float *>(alloc(nw * 4));
    b_[l] = static_cast<float *>(alloc(dout_[l] * 4));
    mw_[l] = static_cast<float *>(alloc(nw * 4));
    vw_[l] = static_cast<float *>(alloc(nw * 4));
    mb_[l] = static_cast<float *>(alloc(dout_[l] * 4));
    vb_[l] = static_cast<float *>(alloc(dout_[l] * 4));
    wimg_[l] = static_cast<uint8_t *>(alloc(static_cast<size_t>(dout_[l]) * ((din_[l] + 63) / 64) * 128));
    wpack_[l] = static_cast<uint8_t *>(alloc(nw * 2));
    ck(cudaMemcpyAsync(w_[l], w.data(), nw * 4, cudaMemcpyHostToDevice, stream_), "upload weights");
    ck(cudaMemcpyAsync(b_[l], b.data(), dout_[l] * 4, cudaMemcpyHostToDevice, stream_), "upload bias");
    ck(cudaStreamSynchronize(stream_), "upload weights");
  }
  void *p = nullptr;
  ck(cudaMalloc(&p, sizeof(double)), "loss");
  allocs_.push_back(p);
  loss_ = static_cast<double *>(p);
  ck(cudaMalloc(&p, sizeof(int)), "err");
  ck(cudaMemsetAsync(p, 0, sizeof(int), stream_), "err");
  allocs_.push_back(p);
  err_ = static_cast<int *>(p);
  for (int q = 0; q < kSurIn; ++q) {
    in_mu[q] = 0.f;
    in_sig[q] = 1.f;
  }
  for (int q = 0; q < kSurOut; ++q) out_s[q] = out_c[q] = 1.f;
  upload_chem();
  pack();
}

Surrogate::~Surrogate() {
  cudaSetDevice(device_);
  for (void *p : allocs_) cudaFree(p);
  free_batch();
  cudaFree(states_);
  cudaFree(labels_);
  cudaFree(x_);
  cudaFree(t_);
  cudaStreamDestroy(stream_);
}

// Stream-ordered: a copy on the legacy default stream from pageable memory
// may still be in flight when a kernel on this non-blocking stream starts.
void Surrogate::upload_chem() {
  ck(cudaMemcpyToSymbolAsync(cP, &chem_, sizeof(DevParams), 0, cudaMemcpyHostToDevice, stream_), "upload mechanism");
  const sur::JudgeTables jt = sur::make_judge_tables(chem_);
  ck(cudaMemcpyToSymbolAsync(sur::cJ, &jt, sizeof(jt), 0, cudaMemcpyHostToDevice, stream_), "upload judge tables");
  ck(cudaStreamSynchronize(stream_), "upload judge tables");
}

void Surrogate::pack() {
  for (int l = 0; l < kSurLayers; ++l) {
    const int64_t nw = static_cast<int64_t>(dout_[l]) * din_[l];
    k_pack<<<(nw + 255) / 256, 256, 0, stream_>>>(w_[l], dout_[l], din_[l], wimg_[l], wpack_[l]);
  }
  ck(cudaGetLastError(), "pack weights");
  packed_ = true;
}

void Surrogate::launch_label(const double *states, double *dy, int64_t n) {
  const size_t smem = 2 * static_cast<size_t>(chem_.nr) * 128 * sizeof(double);  // two rates per reaction and thread
  auto *fn = mech::matches<mech::H2O2>(chem_) ? k_label<mech::H2O2> : k_label<void>;
  ck(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)), "smem");
  fn<<<(n + 127) / 128, 128, smem, stream_>>>(states, dy, n);
  ck(cudaGetLastError(), "label launch");
}

void Surrogate::generate(int64_t n, uint64_t seed, const DevBlock *field, double field_fraction) {
  if (n <= 0) throw std::runtime_error("number of samples must be positive");
  ck(cudaSetDevice(device_), "cudaSetDevice");
  upload_chem();
  cudaFree(states_);
  cudaFree(labels_);
  cudaFree(x_);
  cudaFree(t_);
  states_ = nullptr;
  labels_ = nullptr;
  x_ = nullptr;
  t_ = nullptr;
  ck(cudaMalloc(&states_, n * kSurIn * sizeof(double)), "cudaMalloc samples");
  ck(cudaMalloc(&labels_, n * NS * sizeof(double)), "cudaMalloc labels");
  ck(cudaMalloc(&x_, n * kSurInPad * sizeof(uint16_t)), "cudaMalloc features");
  ck(cudaMalloc(&t_, n * kSurOutPad * sizeof(float)), "cudaMalloc targets");
  n_ = n;
  DevBlock F{};
  if (field) F = *field;
  k_sample<<<(n + 255) / 256, 256, 0, stream_>>>(states_, n, seed, F, field ? 1 : 0, field_fraction, gate);
  ck(cudaGetLastError(), "sample launch");
  launch_label(states_, labels_, n);
  // normalisation from the data
  DevTemp<double> acc(2 * kSurIn + kSurOut, "cudaMalloc stats");
  ck(cudaMemsetAsync(acc.p, 0, (2 * kSurIn + kSurOut) * sizeof(double), stream_), "memset stats");
  k_stats<<<1184, 256, 0, stream_>>>(states_, labels_, n, acc.p);
  double h[2 * kSurIn + kSurOut];
  ck(cudaMemcpyAsync(h, acc.p, sizeof(h), cudaMemcpyDeviceToHost, stream_), "stats copy");
  ck(cudaStreamSynchronize(stream_), "generate");
  Norm nm{};
  for (int q = 0; q < kSurIn; ++q) {
    const double mu = h[q] / n, var = std::max(h[kSurIn + q] / n - mu * mu, 1e-12);
    in_mu[q] = nm.mu[q] = static_cast<float>(mu);
    in_sig[q] = nm.sig[q] = static_cast<float>(std::sqrt(var));
  }
  {
    // target transform from a sub-sample: c_k = median |r_k|, s_k = RMS of
    // asinh(r_k / c_k), r_k = dY_k / (Y_k + eps)
    const int64_t m = std::min<int64_t>(n, 1 << 18);
    std::vector<double> lab(static_cast<size_t>(m) * NS), st(static_cast<size_t>(m) * kSurIn);
    d2h(lab.data(), labels_, lab.size() * 8, "labels copy");
    d2h(st.data(), states_, st.size() * 8, "states copy");
    for (int64_t i = 0; i < m; ++i)
      for (int q = 0; q < NS; ++q) lab[i * NS + q] /= st[i * kSurIn + 2 + q] + kSurYEps;
    // the trust region in dt follows the data (field samples carry the
    // cells' own local time steps)
    double ldt_lo = 1e30, ldt_hi = -1e30;
    for (int64_t i = 0; i < m; ++i) {
      const double l = std::log10(st[i * kSurIn + 11]);
      ldt_lo = std::min(ldt_lo, l);
      ldt_hi = std::max(ldt_hi, l);
    }
    gate.ldt_min = static_cast<float>(ldt_lo - 0.1);
    gate.ldt_max = static_cast<float>(ldt_hi + 0.1);
    for (int q = 0; q < kSurOut; ++q) {
      std::vector<double> a(static_cast<size_t>(m));
      for (int64_t i = 0; i < m; ++i) a[i] = std::fabs(lab[i * NS + q]);
      std::nth_element(a.begin(), a.begin() + m / 2, a.end());
      const double c = std::max(a[m / 2], 1e-14);
      double ss = 0;
      for (int64_t i = 0; i < m; ++i) {
        const double t = std::asinh(lab[i * NS + q] / c);
        ss += t * t;
      }
      out_c[q] = nm.c[q] = static_cast<float>(c);
      out_s[q] = nm.s[q] = static_cast<float>(std::sqrt(ss / m) + 1e-6);
    }
  }
  k_features<<<(n + 255) / 256, 256, 0, stream_>>>(states_, labels_, n, nm, x_, t_);
  ck(cudaGetLastError(), "features launch");
  ck(cudaStreamSynchronize(stream_), "generate");
}

void Surrogate::free_batch() {
  auto free_ = [](auto *&p) {
    cudaFree(p);
    p = nullptr;
  };
  for (int l = 0; l < kSurLayers; ++l) {
    free_(a_[l]);
    free_(dz_[l]);
    free_(part_[l]);
    free_(colsum_[l]);
  }
  for (auto &z : z_) free_(z);
  free_(xb_);
  free_(tb_);
  free_(pred_);
  free_(loss_part_);
  free_(grad_);
  batch_ = 0;
}

void Surrogate::ensure_batch(int batch) {
  if (batch == batch_) return;
  if (batch % mlp::kTile) throw std::runtime_error("batch must be a multiple of 128");
  free_batch();
  const size_t B = static_cast<size_t>(batch), tiles = B / mlp::kTile;
  const int halves = 2 * static_cast<int>(tiles), L = kSurLayers - 1;
  size_t n_param = 0;
  for (int l = 0; l < kSurLayers; ++l) {
    const bool thin = l == 0 || l == L;
    splits_[l] = std::min(halves, thin ? mlp::kSplitThin : mlp::kSplitHidden);
    ck(cudaMalloc(&a_[l], tiles * (l == 0 ? mlp::kChunk : mlp::kTileBytes)), "activations");
    ck(cudaMalloc(&dz_[l], tiles * (l == L ? mlp::kChunk : mlp::kTileBytes)), "output gradients");
    ck(cudaMalloc(&part_[l], static_cast<size_t>(splits_[l]) * kSurHidden * (thin ? 16 : kSurHidden) * 4), "partial");
    ck(cudaMalloc(&colsum_[l], tiles * dout_[l] * 4), "column sums");
    if (l < L) ck(cudaMalloc(&z_[l], B * kSurHidden * 4), "z");
    n_param += static_cast<size_t>(dout_[l]) * din_[l] + dout_[l];
  }
  ck(cudaMalloc(&xb_, B * kSurInPad * 2), "features");
  ck(cudaMalloc(&tb_, B * kSurOutPad * 4), "targets");
  ck(cudaMalloc(&pred_, B * kSurOutPad * 4), "predictions");
  ck(cudaMalloc(&loss_part_, tiles * sizeof(double)), "loss");
  ck(cudaMalloc(&grad_, n_param * 4), "gradients");
  auto smem = [](const void *fn, uint32_t bytes) {
    ck(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)), "smem");
  };
  smem(reinterpret_cast<const void *>(mlp::k_layer<false, true>), mlp::kLayerSmem);
  smem(reinterpret_cast<const void *>(mlp::k_layer<false, false>), mlp::kLayerSmem);
  smem(reinterpret_cast<const void *>(mlp::k_layer<true, true>), mlp::kLayerSmem);
  smem(reinterpret_cast<const void *>(mlp::k_layer<true, false>), mlp::kLayerSmem);
  smem(reinterpret_cast<const void *>(mlp::k_out<true>), mlp::kOutSmem);
  smem(reinterpret_cast<const void *>(mlp::k_out<false>), mlp::kOutSmem);
  smem(reinterpret_cast<const void *>(mlp::k_dw), mlp::kDwSmem);
  batch_ = batch;
}

void Surrogate::gather(const uint16_t *x, const float *t, int64_t n, uint64_t seed, bool in_order) {
  k_gather<<<(batch_ + 127) / 128, 128, 0, stream_>>>(x, t, n, seed, in_order, batch_, a_[0], tb_);
  ck(cudaGetLastError(), "gather");
}

// The hidden layers of the batch in a_[0]: z = a_[l] W_l^T + b_l (kept for
// the backward pass), a_[l + 1] = GELU(z).
void Surrogate::forward(bool keep) {
  const int tiles = batch_ / mlp::kTile;
  for (int l = 0; l < kSurLayers - 1; ++l) {
    auto *fn = l == 0 ? mlp::k_layer<false, true> : mlp::k_layer<false, false>;
    fn<<<tiles, mlp::kThreads, mlp::kLayerSmem, stream_>>>(a_[l], wimg_[l], b_[l], keep ? z_[l] : nullptr, a_[l + 1],
                                                          nullptr, err_);
  }
  ck(cudaGetLastError(), "forward");
}

// The output layer: loss and output gradient of the batch's targets, or the
// predictions.
void Surrogate::output_layer(bool train) {
  const int L = kSurLayers - 1;
  auto *fn = train ? mlp::k_out<true> : mlp::k_out<false>;
  fn<<<batch_ / mlp::kTile, mlp::kTile, mlp::kOutSmem, stream_>>>(a_[L], wimg_[L], b_[L], tb_, batch_, pred_, dz_[L],
                                                                 colsum_[L], loss_part_, err_);
  ck(cudaGetLastError(), "output layer");
}

// Output gradients of every layer down from dz_[L], then the partial weight
// gradients of all layers.
void Surrogate::backward() {
  const int L = kSurLayers - 1;
  for (int l = L; l > 0; --l) {
    auto *fn = l == L ? mlp::k_layer<true, true> : mlp::k_layer<true, false>;
    fn<<<batch_ / mlp::kTile, mlp::kThreads, mlp::kLayerSmem, stream_>>>(dz_[l], wimg_[l], nullptr, z_[l - 1], dz_[l - 1],
                                                                        colsum_[l - 1], err_);
  }
  mlp::DwArgs a{};
  int grid = 0;
  for (int l = 0; l < kSurLayers; ++l) {
    a.p[l] = l == L ? a_[l] : dz_[l];
    a.q[l] = l == L ? dz_[l] : a_[l];
    a.part[l] = part_[l];
    a.splits[l] = splits_[l];
    grid += splits_[l];
  }
  a.halves = 2 * (batch_ / mlp::kTile);
  mlp::k_dw<<<grid, mlp::kThreads, mlp::kDwSmem, stream_>>>(a, err_);
  ck(cudaGetLastError(), "backward");
}

// Sums the partial gradients and the loss, and stores the gradients (grad) or
// takes the Adam step with them.
void Surrogate::reduce(float *grad, double lr, double *loss) {
  mlp::StepArgs a{};
  for (int l = 0; l < kSurLayers; ++l) {
    a.w[l] = w_[l];
    a.b[l] = b_[l];
    a.mw[l] = mw_[l];
    a.vw[l] = vw_[l];
    a.mb[l] = mb_[l];
    a.vb[l] = vb_[l];
    a.img[l] = wimg_[l];
    a.part[l] = part_[l];
    a.colsum[l] = colsum_[l];
    a.splits[l] = splits_[l];
  }
  a.tiles = batch_ / mlp::kTile;
  a.batch = batch_;
  a.loss_part = loss_part_;
  a.loss = loss;
  a.grad = grad;
  a.err = err_;
  a.lr = static_cast<float>(lr);
  a.b1 = 0.9f;
  a.b2 = 0.999f;
  a.eps = 1e-8f;
  a.bc1 = 1.f - std::pow(a.b1, static_cast<float>(adam_t_));
  a.bc2 = 1.f - std::pow(a.b2, static_cast<float>(adam_t_));
  mlp::k_step<<<mlp::kStepBlocks, dim3(32, 8), 0, stream_>>>(a);
  ck(cudaGetLastError(), "gradient step");
}

// Throws if a wait of the kernels since the last check ran out, and starts
// afresh.
void Surrogate::check_waits(const char *what) {
  int err = 0;
  d2h(&err, err_, sizeof(int), "err copy");
  if (!err) return;
  ck(cudaMemsetAsync(err_, 0, sizeof(int), stream_), "err");
  throw std::runtime_error(std::string("tensor-core wait timed out during ") + what);
}

void Surrogate::mark_timeout() {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  ck(cudaMemsetAsync(err_, 1, sizeof(int), stream_), "err");
}

double Surrogate::train(int steps, int batch, double lr, int64_t n_train, float *losses) {
  if (n_ == 0) throw std::runtime_error("generate samples before training");
  if (n_train <= 0 || n_train > n_) n_train = n_;
  ck(cudaSetDevice(device_), "cudaSetDevice");
  ensure_batch(batch);
  // each step's loss stays on the device until the end: no host
  // synchronisation between steps
  DevTemp<double> dloss_buf(static_cast<size_t>(std::max(1, steps)), "cudaMalloc losses");
  double *dloss = dloss_buf.p;
  // all bits set, a NaN that no sum gives: the steps not taken after a timeout
  ck(cudaMemsetAsync(dloss, 0xff, sizeof(double) * static_cast<size_t>(std::max(1, steps)), stream_), "losses");
  const int first = adam_t_;
  for (int s = 0; s < steps; ++s) {
    gather(x_, t_, n_train, mix64(seed_ + 0x5151 * (adam_t_ + 1)), false);
    forward(true);
    output_layer(true);
    backward();
    const double cosine = 0.5 * (1 + std::cos(3.141592653589793 * s / std::max(1, steps)));
    // schedule: cosine decay to 5 % of lr
    const double lr_s = lr * (0.05 + 0.95 * cosine);
    ++adam_t_;
    reduce(nullptr, lr_s, dloss + s);  // new bf16 images too; the inference copy once, below
  }
  pack();
  std::vector<double> hl(static_cast<size_t>(std::max(1, steps)), 0.0);
  cudaError_t st = cudaMemcpyAsync(hl.data(), dloss, sizeof(double) * hl.size(), cudaMemcpyDeviceToHost, stream_);
  if (st == cudaSuccess) st = cudaStreamSynchronize(stream_);
  ck(st, "train steps");
  if (losses)
    for (int s = 0; s < steps; ++s) losses[s] = static_cast<float>(hl[s]);
  int taken = 0;
  for (uint64_t bits = 0; taken < steps; ++taken) {
    std::memcpy(&bits, &hl[taken], sizeof(bits));
    if (bits == ~0ull) break;
  }
  adam_t_ = first + taken;
  check_waits("training");
  return steps > 0 ? hl[steps - 1] : 0.0;
}

std::vector<std::vector<float>> Surrogate::params() const {
  std::vector<std::vector<float>> out;
  for (int l = 0; l < kSurLayers; ++l) {
    std::vector<float> w(static_cast<size_t>(dout_[l]) * din_[l]), b(dout_[l]);
    d2h(w.data(), w_[l], w.size() * 4, "params");
    d2h(b.data(), b_[l], b.size() * 4, "params");
    out.push_back(std::move(w));
    out.push_back(std::move(b));
  }
  return out;
}

void Surrogate::set_params(const std::vector<std::vector<float>> &p) {
  if (p.size() != 2 * kSurLayers) throw std::runtime_error("expected weights and biases of 5 layers");
  for (int l = 0; l < kSurLayers; ++l) {
    if (p[2 * l].size() != static_cast<size_t>(dout_[l]) * din_[l] || p[2 * l + 1].size() != static_cast<size_t>(dout_[l]))
      throw std::runtime_error("parameter shape mismatch");
    ck(cudaMemcpyAsync(w_[l], p[2 * l].data(), p[2 * l].size() * 4, cudaMemcpyHostToDevice, stream_), "set params");
    ck(cudaMemcpyAsync(b_[l], p[2 * l + 1].data(), p[2 * l + 1].size() * 4, cudaMemcpyHostToDevice, stream_),
       "set params");
  }
  pack();
  ck(cudaStreamSynchronize(stream_), "set params");
}

// host states -> features on the device
void Surrogate::features(const double *states_dev, int64_t n, uint16_t *x_dev, float *t_dev, const double *dy_dev) {
  Norm nm{};
  for (int q = 0; q < kSurIn; ++q) {
    nm.mu[q] = in_mu[q];
    nm.sig[q] = in_sig[q];
  }
  for (int q = 0; q < kSurOut; ++q) {
    nm.s[q] = out_s[q];
    nm.c[q] = out_c[q];
  }
  k_features<<<(n + 255) / 256, 256, 0, stream_>>>(states_dev, dy_dev, n, nm, x_dev, t_dev);
  ck(cudaGetLastError(), "features");
}

void Surrogate::label_host(const double *states, int64_t n, double *dy) {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  upload_chem();
  DevTemp<double> s_buf(n * kSurIn, "label alloc"), d_buf(n * NS, "label alloc");
  double *s = s_buf.p, *d = d_buf.p;
  ck(cudaMemcpyAsync(s, states, n * kSurIn * 8, cudaMemcpyHostToDevice, stream_), "label upload");
  launch_label(s, d, n);
  ck(cudaMemcpyAsync(dy, d, n * NS * 8, cudaMemcpyDeviceToHost, stream_), "label download");
  ck(cudaStreamSynchronize(stream_), "label");
}

namespace {
// decode, project and gate the predictions z (batch x 16, bias added)
__global__ void k_decode(const float *z, const double *states, int64_t n, SurrogateDev gd, double *dy,
                         int *accepted) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const double *s = states + i * kSurIn;
  float o[NS];
  for (int k = 0; k < NS; ++k) o[k] = z[i * kSurOutPad + k];
  double d[NS];
  const bool ok = sur::decode<NS>(gd, o, static_cast<float>(s[0]), log10f(static_cast<float>(s[1])),
                                  log10f(static_cast<float>(s[11])), s + 2, d);
  for (int k = 0; k < NS; ++k) dy[i * NS + k] = d[k];
  accepted[i] = ok ? 1 : 0;
}
}  // namespace

void Surrogate::predict_host(const double *states, int64_t n, double *dy, int *accepted) {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  const int batch = static_cast<int>((n + 127) / 128 * 128);
  ensure_batch(batch);
  DevTemp<double> s_buf(static_cast<size_t>(batch) * kSurIn, "predict alloc"), d_buf(n * NS, "predict alloc");
  DevTemp<int> acc_buf(n, "predict alloc");
  double *s = s_buf.p, *d = d_buf.p;
  int *acc = acc_buf.p;
  ck(cudaMemsetAsync(s, 0, static_cast<size_t>(batch) * kSurIn * 8, stream_), "predict memset");
  ck(cudaMemcpyAsync(s, states, n * kSurIn * 8, cudaMemcpyHostToDevice, stream_), "predict upload");
  features(s, n, xb_, nullptr, nullptr);
  gather(xb_, nullptr, n, 0, true);
  forward(false);
  output_layer(false);
  k_decode<<<(n + 255) / 256, 256, 0, stream_>>>(pred_, s, n, device_params(), d, acc);
  ck(cudaGetLastError(), "predict");
  ck(cudaMemcpyAsync(dy, d, n * NS * 8, cudaMemcpyDeviceToHost, stream_), "predict download");
  ck(cudaMemcpyAsync(accepted, acc, n * sizeof(int), cudaMemcpyDeviceToHost, stream_), "predict download");
  ck(cudaStreamSynchronize(stream_), "predict");
  check_waits("prediction");
}

double Surrogate::grad_host(const double *states, const double *dy, int64_t n, std::vector<std::vector<float>> &grads) {
  ck(cudaSetDevice(device_), "cudaSetDevice");
  if (n % 128) throw std::runtime_error("gradient batch must be a multiple of 128");
  const int batch = static_cast<int>(n);
  ensure_batch(batch);
  DevTemp<double> s_buf(n * kSurIn, "grad alloc"), d_buf(n * NS, "grad alloc");
  double *s = s_buf.p, *d = d_buf.p;
  ck(cudaMemcpyAsync(s, states, n * kSurIn * 8, cudaMemcpyHostToDevice, stream_), "grad upload");
  ck(cudaMemcpyAsync(d, dy, n * NS * 8, cudaMemcpyHostToDevice, stream_), "grad upload");
  features(s, n, xb_, tb_, d);
  gather(xb_, nullptr, n, 0, true);
  forward(true);
  output_layer(true);
  backward();
  reduce(grad_, 0.0, loss_);
  grads.assign(2 * kSurLayers, {});
  size_t off = 0;
  for (int l = 0; l < kSurLayers; ++l) {
    grads[2 * l].resize(static_cast<size_t>(dout_[l]) * din_[l]);
    grads[2 * l + 1].resize(dout_[l]);
    for (int q = 2 * l; q < 2 * l + 2; ++q) {
      ck(cudaMemcpyAsync(grads[q].data(), grad_ + off, grads[q].size() * 4, cudaMemcpyDeviceToHost, stream_), "grad copy");
      off += grads[q].size();
    }
  }
  double loss = 0;
  ck(cudaMemcpyAsync(&loss, loss_, sizeof(double), cudaMemcpyDeviceToHost, stream_), "loss");
  ck(cudaStreamSynchronize(stream_), "grad");
  check_waits("the gradients");
  return loss;
}

// Relative errors are taken over samples whose EPI increment reaches 1e-6 in
// some species: below that the chemistry changes nothing the solver resolves,
// and the gate bounds the network's increment by rel_max (Y_k + y_floor).
constexpr double kRelFloor = 1e-6;

SurrogateEval Surrogate::evaluate(int64_t begin, int64_t count) {
  if (begin < 0 || count <= 0 || begin + count > n_) throw std::runtime_error("evaluation range outside the data set");
  std::vector<double> st(count * kSurIn), lab(count * NS), pred(count * NS);
  std::vector<int> acc(count);
  d2h(st.data(), states_ + begin * kSurIn, st.size() * 8, "eval copy");
  d2h(lab.data(), labels_ + begin * NS, lab.size() * 8, "eval copy");
  const int64_t chunk = 1 << 18;
  for (int64_t q = 0; q < count; q += chunk) {
    const int64_t m = std::min(chunk, count - q);
    predict_host(st.data() + q * kSurIn, m, pred.data() + q * NS, acc.data() + q);
  }
  SurrogateEval e{};
  e.count = count;
  double rel_sum = 0;
  int64_t rel_n = 0, n_acc = 0;
  std::vector<double> rel_all;
  rel_all.reserve(static_cast<size_t>(count));
  for (int64_t i = 0; i < count; ++i) {
    double nrm = 0, err = 0, abs_sum = 0;
    bool finite = true;
    for (int k = 0; k < NS; ++k) {
      const double d = pred[i * NS + k] - lab[i * NS + k];
      finite = finite && std::isfinite(d);
      nrm = std::max(nrm, std::fabs(lab[i * NS + k]));
      err = std::max(err, std::fabs(d));
      abs_sum += std::fabs(d);
    }
    if (!finite) {
      ++e.nonfinite;
      if (nrm > kRelFloor) rel_all.push_back(std::numeric_limits<double>::infinity());
      continue;
    }
    const double r = nrm > kRelFloor ? err / nrm : -1;
    if (r >= 0) rel_all.push_back(r);
    if (!acc[i]) continue;
    ++n_acc;
    e.mean_abs += abs_sum / NS;
    if (r >= 0) {
      rel_sum += r;
      ++rel_n;
      e.max_rel = std::max(e.max_rel, r);
    }
    double dmax = 0;
    for (int el = 0; el < n_elem_; ++el) {
      double defect = 0, total = 0;
      for (int k = 0; k < NS; ++k) {
        const double a = elem_comp_[k * n_elem_ + el] / chem_.mw[k];
        defect += a * pred[i * NS + k];
        total += a * st[i * kSurIn + 2 + k];
      }
      if (total > 0) dmax = std::max(dmax, std::fabs(defect) / total);
    }
    e.max_defect = std::max(e.max_defect, dmax);
    e.mean_defect += dmax;
  }
  e.gate_pass = static_cast<double>(n_acc) / static_cast<double>(count);
  e.mean_rel = rel_n ? rel_sum / rel_n : 0;
  e.rel_count = rel_n;
  if (n_acc) {
    e.mean_abs /= n_acc;
    e.mean_defect /= n_acc;
  }
  if (!rel_all.empty()) {
    auto at = [&](double q) {
      const size_t k = static_cast<size_t>(q * (rel_all.size() - 1));
      std::nth_element(rel_all.begin(), rel_all.begin() + k, rel_all.end());
      return rel_all[k];
    };
    e.median_rel_all = at(0.5);
    e.p90_rel_all = at(0.9);
  }
  return e;
}

const SurrogateDev &Surrogate::device_params() {
  for (int l = 0; l < kSurLayers; ++l) {
    dev_.w_packed[l] = wpack_[l];
    dev_.bias[l] = b_[l];
  }
  for (int q = 0; q < kSurIn; ++q) {
    dev_.in_mu[q] = in_mu[q];
    dev_.in_sig[q] = in_sig[q];
  }
  for (int q = 0; q < kSurOut; ++q) {
    dev_.out_s[q] = out_s[q];
    dev_.out_c[q] = out_c[q];
  }
  dev_.n_elem = n_elem_;
  for (int e = 0; e < kMaxElem * kMaxSpec; ++e) dev_.elem[e] = 0.f;
  for (int e = 0; e < n_elem_; ++e)
    for (int k = 0; k < NS; ++k) dev_.elem[e * kMaxSpec + k] = static_cast<float>(elem_comp_[k * n_elem_ + e] / chem_.mw[k]);
  dev_.gate = gate;
  return dev_;
}

void Surrogate::save(const std::string &path) const {
  std::ofstream f(path, std::ios::binary);
  if (!f) throw std::runtime_error("cannot write " + path);
  const char magic[8] = {'O', 'S', 'T', 'C', 'M', 'L', 'P', '5'};
  f.write(magic, 8);
  f.write(reinterpret_cast<const char *>(in_mu.data()), sizeof(in_mu));
  f.write(reinterpret_cast<const char *>(in_sig.data()), sizeof(in_sig));
  f.write(reinterpret_cast<const char *>(out_c.data()), sizeof(out_c));
  f.write(reinterpret_cast<const char *>(out_s.data()), sizeof(out_s));
  f.write(reinterpret_cast<const char *>(&gate), sizeof(gate));
  for (const auto &p : params()) f.write(reinterpret_cast<const char *>(p.data()), p.size() * 4);
}

void Surrogate::load(const std::string &path) {
  std::ifstream f(path, std::ios::binary);
  if (!f) throw std::runtime_error("cannot open " + path);
  char magic[8];
  f.read(magic, 8);
  if (std::memcmp(magic, "OSTCMLP5", 8) != 0) throw std::runtime_error(path + " is not a surrogate file");
  f.read(reinterpret_cast<char *>(in_mu.data()), sizeof(in_mu));
  f.read(reinterpret_cast<char *>(in_sig.data()), sizeof(in_sig));
  f.read(reinterpret_cast<char *>(out_c.data()), sizeof(out_c));
  f.read(reinterpret_cast<char *>(out_s.data()), sizeof(out_s));
  f.read(reinterpret_cast<char *>(&gate), sizeof(gate));
  auto p = params();
  for (auto &v : p) f.read(reinterpret_cast<char *>(v.data()), v.size() * 4);
  if (!f) throw std::runtime_error(path + " is truncated");
  set_params(p);
}

}  // namespace ostc
