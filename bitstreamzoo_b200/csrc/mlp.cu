// Learned schedule cost model: a small FP32 MLP (in -> H -> H -> H -> 1,
// ReLU) trained and evaluated with hand-written CUDA kernels.
//
// It predicts log(kernel time) from DAG features plus a candidate schedule;
// the autotuner uses it to pick a schedule without timing every candidate.
// The network is small (hidden 256, a few hundred rows), so the kernels are
// plain SIMT FFMA and every product is bound by latency, not by its
// arithmetic:
//   * gemm: C[M,N] = op(A)[M,K] * op(B)[K,N] (+ bias, ReLU) with 32x32 output
//     tiles (64 blocks for 256 x 256; 64x64 tiles ran on 16 of 148 SMs), K in
//     chunks of 256 loaded at once, each of the 8 warps summing an eighth of
//     the chunk, and one sum over the warps at the end.  op() = transpose
//     flags, which give both backward products without materializing
//     transposes; the ReLU's backward mask and the bias gradients (column
//     sums) are part of the products that read the same data;
//   * mse (loss + gradient), Adam (one fused update over the flat parameter
//     vector).
// Loss, gradients and predictions of 256 rows on a B200: 675 us a call with
// 64x64 tiles and kernels of their own for masks and column sums, 225 us so;
// see gradients() and predict().
// Parameters live in one flat device array: W1 b1 W2 b2 ... Wout bout, each
// W stored row-major [fan_in, fan_out].
#include "mlp.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "device.h"
#include "pdl.cuh"

namespace bsz {
namespace {

constexpr int kTile = 32;           // output tile, both ways
constexpr int kChunk = 256;         // K per load
constexpr int kPad = kTile + 4;     // row stride in shared memory: 16-byte aligned rows
constexpr int kGemmWarps = 8;
constexpr size_t kGemmSmem = 2 * sizeof(float) * kChunk * kPad;

// A [rows x kc] piece of X into S[k][row]: rows r0.., k from k0.  T: X is
// [K, R] (k slow), else [R, K].  Eight loads of each thread are in flight at a
// time (a load and its store in turn made a product of 256 x 256 x 256 take
// 11 to 18 us, 4 us so); 16-byte loads where rows allow them.
template <int T>
__device__ __forceinline__ void load_piece(float* S, const float* __restrict__ X, int R, int K, int r0, int k0, int kc) {
  constexpr int kBatch = 8, kThreads = kGemmWarps * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool vec = ((T ? R : K) & 3) == 0 && (k0 & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  if (vec) {
    float4 v[kBatch];
    if (T) {
      for (int i0 = threadIdx.x; i0 < kc * (kTile / 4); i0 += kBatch * kThreads) {
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int i = i0 + j * kThreads, k = i >> 3, r = r0 + (i & 7) * 4;
          v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (k < kc && r < R) v[j] = *reinterpret_cast<const float4*>(X + (size_t)(k0 + k) * R + r);
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int i = i0 + j * kThreads, k = i >> 3;
          if (k < kc) *reinterpret_cast<float4*>(S + k * kPad + (i & 7) * 4) = v[j];
        }
      }
    } else {
      // 16 rows x 8 k per warp: one sector a row, and the transposed stores
      // meet no bank conflict
      const int r = (lane & 15) + 16 * (warp & 1), kq = (lane >> 4) * 4 + 8 * (warp >> 1);
      for (int b = 0; b < kc; b += 8 * (kGemmWarps / 2) * kBatch) {
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int k = b + j * 8 * (kGemmWarps / 2) + kq;
          v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (k < kc && r0 + r < R) v[j] = *reinterpret_cast<const float4*>(X + (size_t)(r0 + r) * K + k0 + k);
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int k = b + j * 8 * (kGemmWarps / 2) + kq;
          if (k < kc) {
            S[k * kPad + r] = v[j].x;
            S[(k + 1) * kPad + r] = v[j].y;
            S[(k + 2) * kPad + r] = v[j].z;
            S[(k + 3) * kPad + r] = v[j].w;
          }
        }
      }
    }
    return;
  }
  for (int i0 = threadIdx.x; i0 < kc * kTile; i0 += kBatch * kThreads) {
    float v[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int i = i0 + j * kThreads;
      const int k = T ? i / kTile : i % kc, r = T ? i % kTile : i / kc;
      v[j] = 0.f;
      if (i < kc * kTile && r0 + r < R) v[j] = T ? X[(size_t)(k0 + k) * R + r0 + r] : X[(size_t)(r0 + r) * K + k0 + k];
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int i = i0 + j * kThreads;
      const int k = T ? i / kTile : i % kc, r = T ? i % kTile : i / kc;
      if (i < kc * kTile) S[k * kPad + r] = v[j];
    }
  }
}

// C = op(A) * op(B) (+ bias[N]) (ReLU).  A is [M,K] (TA=0) or [K,M] (TA=1);
// B is [K,N] (TB=0) or [N,K] (TB=1).  All row-major.  mask: C is zeroed where
// mask[m,n] <= 0.  colsum: also sum_k op(B)[k,n] into colsum[n].
template <int TA, int TB>
__global__ void __launch_bounds__(kGemmWarps * 32)
k_gemm(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
       const float* __restrict__ bias, const float* __restrict__ mask, float* __restrict__ colsum, int M, int N, int K,
       int relu) {
  after_previous(A, B, bias, mask);
  extern __shared__ __align__(16) float s_mem[];
  float* As = s_mem;
  float* Bs = s_mem + kChunk * kPad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = blockIdx.x * kTile, n0 = blockIdx.y * kTile;
  const int tm = (lane >> 2) * 4, tn = (lane & 3) * 8;   // this lane's 4 x 8 outputs
  const bool sums = colsum != nullptr && blockIdx.x == 0;
  float acc[4][8] = {};
  float cs = 0.f;
  for (int k0 = 0; k0 < K; k0 += kChunk) {
    const int kc = min(kChunk, K - k0);
    if (k0) __syncthreads();
    load_piece<TA>(As, A, M, K, m0, k0, kc);
    load_piece<!TB>(Bs, B, N, K, n0, k0, kc);
    __syncthreads();
    const int per = (kc + kGemmWarps - 1) / kGemmWarps;
    const int k_end = min(kc, (warp + 1) * per);
#pragma unroll 4
    for (int k = warp * per; k < k_end; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(As + k * kPad + tm);
      const float4 b0 = *reinterpret_cast<const float4*>(Bs + k * kPad + tn);
      const float4 b1 = *reinterpret_cast<const float4*>(Bs + k * kPad + tn + 4);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      if (sums) cs += Bs[k * kPad + lane];
    }
  }
  // sum over the warps, in warp order
  __syncthreads();
  float* part = s_mem;   // [warp][32][32]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      *reinterpret_cast<float4*>(part + (warp * kTile + tm + i) * kTile + tn + j) =
          make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  float* part_cs = part + kGemmWarps * kTile * kTile;
  if (sums) part_cs[warp * kTile + lane] = cs;
  __syncthreads();
  for (int r = warp; r < kTile; r += kGemmWarps) {
    const int m = m0 + r, n = n0 + lane;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kGemmWarps; ++w) v += part[(w * kTile + r) * kTile + lane];
    if (m >= M || n >= N) continue;
    if (bias) v += bias[n];
    if (relu) v = fmaxf(v, 0.f);
    if (mask && mask[(size_t)m * N + n] <= 0.f) v = 0.f;
    C[(size_t)m * N + n] = v;
  }
  if (sums && warp == 0 && n0 + lane < N) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kGemmWarps; ++w) v += part_cs[w * kTile + lane];
    colsum[n0 + lane] = v;
  }
}
static_assert(sizeof(float) * (kGemmWarps * kTile * kTile + kGemmWarps * kTile) <= kGemmSmem, "the sums reuse the tiles");

// loss = mean((p - t)^2), dp = 2 (p - t) / n
__global__ void k_mse(const float* __restrict__ p, const float* __restrict__ t, float* __restrict__ dp,
                      float* __restrict__ loss, int n) {
  after_previous(p, t);
  __shared__ float part[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    float e = p[i] - t[i];
    s += e * e;
    if (dp) dp[i] = 2.f * e / n;
  }
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = part[0] / n;
}

__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int64_t n, float lr, float b1, float b2, float eps,
                       float c1, float c2, float wd) {
  after_previous(w, g, m, v);
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gi = g[i];
  float mi = b1 * m[i] + (1.f - b1) * gi;
  float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  // decoupled weight decay (AdamW): w <- w - lr * (mhat / (sqrt(vhat) + eps) + wd * w)
  w[i] -= lr * ((mi / c1) / (sqrtf(vi / c2) + eps) + wd * w[i]);
}

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

template <int TA, int TB>
void gemm(cudaStream_t s, const float* A, const float* B, float* C, const float* bias, const float* mask,
          float* colsum, int M, int N, int K, int relu) {
  // rows along x: a grid has 65,535 blocks along y, two million rows
  dim3 grid((M + kTile - 1) / kTile, (N + kTile - 1) / kTile);
  launch_after(s, grid, kGemmWarps * 32, kGemmSmem, k_gemm<TA, TB>, A, B, C, bias, mask, colsum, M, N, K, relu);
  check(cudaGetLastError(), "mlp gemm launch");
}

// Per device: the products' shared-memory size.
void set_gemm_attrs() {
  check(cudaFuncSetAttribute(k_gemm<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem), "mlp attr");
  check(cudaFuncSetAttribute(k_gemm<1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem), "mlp attr");
  check(cudaFuncSetAttribute(k_gemm<0, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem), "mlp attr");
}

}  // namespace

Mlp::Mlp(int in_dim, int hidden, int layers, uint64_t seed, Device& dev) : dev_(dev), stream_(dev.stream()) {
  if (in_dim < 1 || hidden < 1 || layers < 1) throw std::invalid_argument("mlp: bad shape");
  set_gemm_attrs();
  dims_.push_back(in_dim);
  for (int l = 0; l < layers; ++l) dims_.push_back(hidden);
  dims_.push_back(1);
  for (size_t l = 0; l + 1 < dims_.size(); ++l) {
    woff_.push_back(n_params_);
    n_params_ += static_cast<int64_t>(dims_[l]) * dims_[l + 1];
    boff_.push_back(n_params_);
    n_params_ += dims_[l + 1];
  }
  // He initialisation, zero biases
  std::vector<float> h(n_params_, 0.f);
  std::mt19937_64 rng(seed);
  for (size_t l = 0; l + 1 < dims_.size(); ++l) {
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / dims_[l]));
    for (int64_t i = 0; i < static_cast<int64_t>(dims_[l]) * dims_[l + 1]; ++i) h[woff_[l] + i] = nd(rng);
  }
  const size_t bytes = static_cast<size_t>(n_params_) * 4;
  check(cudaMalloc(&w_, bytes), "mlp alloc");
  check(cudaMalloc(&g_, bytes), "mlp alloc");
  check(cudaMalloc(&m_, bytes), "mlp alloc");
  check(cudaMalloc(&v_, bytes), "mlp alloc");
  check(cudaMalloc(&loss_, 256), "mlp alloc");
  check(cudaMemcpyAsync(w_, h.data(), bytes, cudaMemcpyHostToDevice, stream_), "mlp init");
  check(cudaMemsetAsync(m_, 0, bytes, stream_), "mlp init");
  check(cudaMemsetAsync(v_, 0, bytes, stream_), "mlp init");
  check(cudaStreamSynchronize(stream_), "mlp init");
}

Mlp::~Mlp() {
  cudaStreamSynchronize(stream_);
  for (float* p : {w_, g_, m_, v_, x_, y_, loss_}) if (p) cudaFree(p);
  for (float* p : act_) cudaFree(p);
  for (float* p : delta_) cudaFree(p);
}

void Mlp::ensure(int n) {
  if (n <= cap_) return;
  cudaStreamSynchronize(stream_);
  for (float* p : act_) cudaFree(p);
  for (float* p : delta_) cudaFree(p);
  if (x_) cudaFree(x_);
  if (y_) cudaFree(y_);
  x_ = y_ = nullptr;
  act_.clear();
  delta_.clear();
  cap_ = std::max(n, 256);
  check(cudaMalloc(&x_, static_cast<size_t>(cap_) * dims_[0] * 4), "mlp alloc");
  check(cudaMalloc(&y_, static_cast<size_t>(cap_) * 4), "mlp alloc");
  for (size_t l = 1; l < dims_.size(); ++l) {
    float *a = nullptr, *d = nullptr;
    check(cudaMalloc(&a, static_cast<size_t>(cap_) * dims_[l] * 4), "mlp alloc");
    check(cudaMalloc(&d, static_cast<size_t>(cap_) * dims_[l] * 4), "mlp alloc");
    act_.push_back(a);
    delta_.push_back(d);
  }
}

// Rows, targets and results of a call pass through a page-locked block while
// they are small: a copy from or into the caller's pageable memory by the
// driver takes several times as long.  The block comes from the device's pool
// and goes back when the call, which waits for its results, returns: one of the
// model's own took its first call 2.5 ms to allocate.  Past kMaxBlock the
// device's ring of copy buffers does it, whose size does not follow the rows'.
constexpr size_t kMaxBlock = size_t(4) << 20;

Mlp::Block Mlp::upload(const float* x, const float* y, int n) {
  ensure(n);
  const size_t results = 1 + std::max<size_t>(static_cast<size_t>(n_params_), static_cast<size_t>(n));
  const size_t nx = static_cast<size_t>(n) * dims_[0], ny = y ? static_cast<size_t>(n) : 0;
  const bool small = 4 * (results + nx + ny) <= kMaxBlock;
  Block b;
  b.mem = dev_.pinned_block(small ? 4 * (results + nx + ny) : 4);
  b.loss = static_cast<float*>(b.mem.get());
  if (!small) {
    dev_.h2d(x_, x, nx * 4);
    dev_.h2d(y_, y, ny * 4);
    return b;
  }
  b.out = b.loss + 1;
  float* h = b.loss + results;
  std::memcpy(h, x, nx * 4);
  check(cudaMemcpyAsync(x_, h, nx * 4, cudaMemcpyHostToDevice, stream_), "mlp upload");
  if (y) {
    std::memcpy(h + nx, y, ny * 4);
    check(cudaMemcpyAsync(y_, h + nx, ny * 4, cudaMemcpyHostToDevice, stream_), "mlp upload");
  }
  return b;
}

void Mlp::download(const Block& b, float* dst, const float* src, size_t n) {
  if (!b.out) {
    dev_.d2h(dst, src, n * 4);
    check(cudaStreamSynchronize(stream_), "mlp download");
    return;
  }
  check(cudaMemcpyAsync(b.out, src, n * 4, cudaMemcpyDeviceToHost, stream_), "mlp download");
  check(cudaStreamSynchronize(stream_), "mlp download");
  std::memcpy(dst, b.out, n * 4);
}

void Mlp::forward(int n) {
  const int L = static_cast<int>(dims_.size()) - 1;
  for (int l = 0; l < L; ++l) {
    const float* in = l == 0 ? x_ : act_[l - 1];
    gemm<0, 0>(stream_, in, w_ + woff_[l], act_[l], w_ + boff_[l], nullptr, nullptr, n, dims_[l + 1], dims_[l],
               l + 1 < L ? 1 : 0);
    ++launches;
  }
}

void Mlp::backward(int n, float* loss) {
  const int L = static_cast<int>(dims_.size()) - 1;
  launch_after(stream_, 1, 256, 0, k_mse, act_[L - 1], y_, delta_[L - 1], loss_, n);
  check(cudaGetLastError(), "mlp mse");
  for (int l = L - 1; l >= 0; --l) {
    const float* in = l == 0 ? x_ : act_[l - 1];
    // dW_l = in^T * delta_l ; db_l = colsum(delta_l)
    gemm<1, 0>(stream_, in, delta_[l], g_ + woff_[l], nullptr, nullptr, g_ + boff_[l], dims_[l], dims_[l + 1], n, 0);
    ++launches;
    if (l > 0) {
      // delta_{l-1} = (delta_l * W_l^T) .* relu'(act_{l-1})
      gemm<0, 1>(stream_, delta_[l], w_ + woff_[l], delta_[l - 1], nullptr, act_[l - 1], nullptr, n, dims_[l],
                 dims_[l + 1], 0);
      ++launches;
    }
  }
  ++launches;
  check(cudaMemcpyAsync(loss, loss_, 4, cudaMemcpyDeviceToHost, stream_), "mlp loss");
}

float Mlp::train_step(const float* x, const float* y, int n, float lr) {
  const Block block = upload(x, y, n);
  forward(n);
  backward(n, block.loss);
  check(cudaStreamSynchronize(stream_), "mlp backward");
  const float loss = *block.loss;
  ++step_;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, static_cast<float>(step_));
  const float c2 = 1.f - std::pow(b2, static_cast<float>(step_));
  launch_after(stream_, static_cast<unsigned>((n_params_ + 255) / 256), 256, 0, k_adam, w_, g_, m_, v_, n_params_, lr,
               b1, b2, 1e-8f, c1, c2, weight_decay_);
  check(cudaGetLastError(), "mlp adam");
  ++launches;
  return loss;
}

void Mlp::predict(const float* x, int n, float* out) {
  const Block block = upload(x, nullptr, n);
  forward(n);
  download(block, out, act_.back(), static_cast<size_t>(n));
}

float Mlp::gradients(const float* x, const float* y, int n, float* grad) {
  const Block block = upload(x, y, n);
  forward(n);
  backward(n, block.loss);
  download(block, grad, g_, static_cast<size_t>(n_params_));
  return *block.loss;
}

void Mlp::get_params(float* out) const {
  check(cudaStreamSynchronize(stream_), "mlp params");
  check(cudaMemcpy(out, w_, static_cast<size_t>(n_params_) * 4, cudaMemcpyDeviceToHost), "mlp params");
}

void Mlp::set_params(const float* in) {
  check(cudaMemcpyAsync(w_, in, static_cast<size_t>(n_params_) * 4, cudaMemcpyHostToDevice, stream_),
        "mlp params");
  check(cudaMemsetAsync(m_, 0, static_cast<size_t>(n_params_) * 4, stream_), "mlp params");
  check(cudaMemsetAsync(v_, 0, static_cast<size_t>(n_params_) * 4, stream_), "mlp params");
  check(cudaStreamSynchronize(stream_), "mlp params");
  step_ = 0;
}

}  // namespace bsz
