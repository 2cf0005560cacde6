// Logistic-regression log-density + gradient in FP32 for 129 to 256 features:
// Z on the CUDA cores, X^T R on the tensor cores.
//
// Mathematics as in logreg_simt.cu.  Three launches before the reduction:
//   states    Q^T [features][chains], zero-padded, so that
//   products  a CTA (128 threads, 8 rows x 8 chains each) forms Z of 128 rows x
//             64 chains from X^T and Q^T, 16 features a stage, four stages of
//             16-byte asynchronous copies; then the log-likelihood sums and the
//             residuals, FP16 hi + lo, to memory [rows][chains], scaled by a power
//             of two of the largest of a chain's 32 (rows that are all but
//             fitted leave residuals far below FP16's range);
//   gradient  grad_tc.cuh.
// Z is one chain of FMAs in ascending features and the log-likelihood is added by
// fours of rows in FP32, then in float64: logreg_simt.cu's bits.
//
// What bounds it: FMA issue of the products (an 8 x 8 thread's shared loads take
// as long as its FMAs: 107 of 128 FMAs a clock and SM).  30,011 x 237, 192 chains:
// 359 us an evaluation by logreg_simt.cu (4 x 4 a thread, unpipelined, G on the
// CUDA cores), 106 so: products 63, gradient 25, reduction 10; 300 x 130, 16 chains
// 61 and 38.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>

#include "engine.h"
#include "grad_tc.cuh"
#include "split_reduce.cuh"

namespace gbm {
namespace {

constexpr int kWideRT = 128, kWideCT = 64, kWideK = 16, kWideRing = 4;
constexpr int kWideThreads = 128;
constexpr int kWideStage = kWideK * (kWideRT + kWideCT);          // floats
constexpr int kWideSmem = kWideRing * kWideStage * 4;
static_assert(kWideSmem >= 16 * kWideCT * 8, "likelihood sums fit the stages");

__device__ __forceinline__ void wide_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// X [N][D] -> X^T [Dp][Np], zero-padded; ym = y - 1/2 (zero past N).
__global__ void wide_pack_kernel(const float* __restrict__ X, const float* __restrict__ y,
                                 int64_t N, int64_t Np, int D, int Dp, float* __restrict__ xt,
                                 float* __restrict__ ym) {
  __shared__ float t[32][33];
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int d0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int64_t r = r0 + i;
    const int d = d0 + threadIdx.x;
    t[i][threadIdx.x] = (r < N && d < D) ? X[r * D + d] : 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y)
    if (d0 + i < Dp) xt[(size_t)(d0 + i) * Np + r0 + threadIdx.x] = t[threadIdx.x][i];
  if (blockIdx.y == 0 && threadIdx.y == 0) {
    const int64_t r = r0 + threadIdx.x;
    ym[r] = r < N ? y[r] - 0.5f : 0.f;
  }
}

// Q [n][ldq] -> Q^T [Dp][cp], zero outside (n, D).
__global__ void wide_states_kernel(const float* __restrict__ Q, int ldq,
                                   const int* __restrict__ n_dev, int c_base, int c_lim, int D,
                                   int Dp, int cp, float* __restrict__ qt) {
  __shared__ float t[32][33];
  const int n = chunk_count(*n_dev, c_base, c_lim);
  const int c0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, d = d0 + threadIdx.x;
    t[i][threadIdx.x] = (c < n && d < D) ? Q[(size_t)c * ldq + d] : 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y)
    if (d0 + i < Dp) qt[(size_t)(d0 + i) * cp + c0 + threadIdx.x] = t[threadIdx.x][i];
}

__global__ void __launch_bounds__(kWideThreads, 3)
wide_products_kernel(const float* __restrict__ xt, int64_t Np, const float* __restrict__ y,
                     int N, int Dp, const float* __restrict__ qt, int cp,
                     const int* __restrict__ n_dev, int c_base, int c_lim,
                     double* __restrict__ lpart, __half* __restrict__ rhi,
                     __half* __restrict__ rlo, float* __restrict__ rscale) {
  extern __shared__ __align__(16) float stages[];
  const int n = chunk_count(*n_dev, c_base, c_lim);
  const int c0 = blockIdx.x * kWideCT;
  if (c0 >= n) return;
  const int64_t r0 = (int64_t)blockIdx.y * kWideRT;
  const int tid = threadIdx.x, lane = tid & 31;
  // A warp has 32 rows: this thread's are ry.. and ry + 16..
  const int ty = (tid >> 5) * 4 + (lane >> 3), ry = (tid >> 5) * 32 + (lane >> 3) * 4;
  const int tx = lane & 7;                       // chains 4 tx.., 32 + 4 tx..
  const float* xsrc = xt + r0;
  const float* qsrc = qt + c0;
  const int chunks = Dp / kWideK;
  auto copy = [&](int ch) {
    if (ch < chunks) {
      float* st = stages + (ch % kWideRing) * kWideStage;
#pragma unroll
      for (int i = 0; i < kWideK * kWideRT / 4 / kWideThreads; ++i) {
        const int e = tid + i * kWideThreads, k = e / (kWideRT / 4), r = e % (kWideRT / 4) * 4;
        wide_copy16(st + k * kWideRT + r, xsrc + (size_t)(ch * kWideK + k) * Np + r);
      }
#pragma unroll
      for (int i = 0; i < kWideK * kWideCT / 4 / kWideThreads; ++i) {
        const int e = tid + i * kWideThreads, k = e / (kWideCT / 4), c = e % (kWideCT / 4) * 4;
        wide_copy16(st + kWideK * kWideRT + k * kWideCT + c,
                    qsrc + (size_t)(ch * kWideK + k) * cp + c);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 z[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) z[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int ch = 0; ch < kWideRing - 1; ++ch) copy(ch);
  for (int ch = 0; ch < chunks; ++ch) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kWideRing - 2) : "memory");
    __syncthreads();   // this stage is complete, the last one is free
    copy(ch + kWideRing - 1);
    const float* xs = stages + (ch % kWideRing) * kWideStage + ry;
    const float* qs = stages + (ch % kWideRing) * kWideStage + kWideK * kWideRT + 4 * tx;
#pragma unroll
    for (int k = 0; k < kWideK; ++k) {
      const float4 x0 = *reinterpret_cast<const float4*>(xs + k * kWideRT);
      const float4 x1 = *reinterpret_cast<const float4*>(xs + k * kWideRT + 16);
      const float4 q0 = *reinterpret_cast<const float4*>(qs + k * kWideCT);
      const float4 q1 = *reinterpret_cast<const float4*>(qs + k * kWideCT + 32);
      const float xa[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
      const float2 qa[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w),
                            make_float2(q1.x, q1.y), make_float2(q1.z, q1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          z[i][j] = __ffma2_rn(make_float2(xa[i], xa[i]), qa[j], z[i][j]);
    }
  }
  // Log-likelihood (by fours of rows in FP32) and residuals, in the place of z.
  double ll[8];
  float most[8];       // largest residual of each chain
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    ll[c] = 0.0;
    most[c] = 0.f;
  }
  constexpr int kTurn = 2;
  float four[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) four[c] = 0.f;
  // Two rows an iteration of a rolled loop, in which z turns: unrolled over its eight
  // rows this runs once, from a cold instruction cache (2000 x 200, 64 chains: 21.7 us
  // for the kernel, 16.9 so).
#pragma unroll 1
  for (int k = 0; k < 8; k += kTurn) {
#pragma unroll
    for (int b = 0; b < kTurn; ++b) {
      const int64_t row = r0 + ry + 16 * (k >> 2) + ((k + b) & 3);
      if (row < N) {
        const float yv = y[row];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float& at = e ? z[b][j].y : z[b][j].x;
            const float zv = at;
            const float t = expf(-fabsf(zv)), l = log1pf(t);
            // bernoulli.py:126-140: -softplus(z) (1 - y) - softplus(-z) y
            const float up = fmaxf(zv, 0.f) + l, down = fmaxf(-zv, 0.f) + l;
            four[2 * j + e] += -up * (1.f - yv) - down * yv;
            // y - sigmoid(z) from w = sigmoid(-|z|): a row that is all but fitted
            // keeps its residual's bits, whichever its label.  1 - v is exact, and
            // better than the product while it has bits enough.
            const float v = tc::rcp_approx(1.f + t);
            const float w = t > 0x1p-7f ? 1.f - v : t * v;
            at = zv >= 0.f ? (yv - 1.f) + w : yv - w;
            most[2 * j + e] = fmaxf(most[2 * j + e], fabsf(at));
          }
        }
      }
    }
    if (((k + kTurn) & 3) == 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        ll[c] += (double)four[c];
        four[c] = 0.f;
      }
    }
    // The rows turn: after eight they are in their places again.
    float2 done[kTurn][4];
#pragma unroll
    for (int b = 0; b < kTurn; ++b)
#pragma unroll
      for (int j = 0; j < 4; ++j) done[b][j] = z[b][j];
#pragma unroll
    for (int m = 0; m < 8 - kTurn; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) z[m][j] = z[m + kTurn][j];
#pragma unroll
    for (int b = 0; b < kTurn; ++b)
#pragma unroll
      for (int j = 0; j < 4; ++j) z[8 - kTurn + b][j] = done[b][j];
  }
  // A chain's 32 residuals are stored as multiples of the power of two that takes
  // the largest of them below 2^15; gradient sums are in multiples of 2^-15.
  float up[8], back[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    most[c] = fmaxf(most[c], __shfl_xor_sync(~0u, most[c], 8));
    most[c] = fmaxf(most[c], __shfl_xor_sync(~0u, most[c], 16));
    const int e = max(float_exponent(__float_as_uint(most[c])), -100);
    up[c] = __int_as_float((kF16Top - e + 127) << 23);
    back[c] = __int_as_float((15 - kF16Top + e + 127) << 23);
  }
  if (lane < 8) {
    float* s = rscale + ((size_t)blockIdx.y * (kWideRT / 32) + (tid >> 5)) * cp + c0 + 4 * tx;
    *reinterpret_cast<float4*>(s) = make_float4(back[0], back[1], back[2], back[3]);
    *reinterpret_cast<float4*>(s + 32) = make_float4(back[4], back[5], back[6], back[7]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t row = r0 + ry + 16 * (i >> 2) + (i & 3);
    if (row < N) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float rx = z[i][j].x * up[2 * j], ry = z[i][j].y * up[2 * j + 1];
        const __half2 a = __floats2half2_rn(rx, ry);
        const float2 af = __half22float2(a);
        const __half2 b = __floats2half2_rn(rx - af.x, ry - af.y);
        hi[j] = *reinterpret_cast<const uint32_t*>(&a);
        lo[j] = *reinterpret_cast<const uint32_t*>(&b);
      }
      const size_t at = (size_t)row * cp + c0 + 4 * tx;
      *reinterpret_cast<uint2*>(rhi + at) = make_uint2(hi[0], hi[1]);
      *reinterpret_cast<uint2*>(rhi + at + 32) = make_uint2(hi[2], hi[3]);
      *reinterpret_cast<uint2*>(rlo + at) = make_uint2(lo[0], lo[1]);
      *reinterpret_cast<uint2*>(rlo + at + 32) = make_uint2(lo[2], lo[3]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();   // every thread is done with the stages
  double* red = reinterpret_cast<double*>(stages);   // [16][64]
#pragma unroll
  for (int c = 0; c < 8; ++c)
    red[ty * kWideCT + (c < 4 ? 4 * tx + c : 32 + 4 * tx + c - 4)] = ll[c];
  __syncthreads();
  if (tid < kWideCT && c0 + tid < n) {
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < 16; ++t) s += red[t * kWideCT + tid];
    lpart[(size_t)blockIdx.y * n + c0 + tid] = s;
  }
}

// Sizes of a target and of its launches.
struct WideShape {
  int64_t N, D;
  int sms;
  struct Layout {
    int64_t cp;                    // chains rounded up to whole tiles
    size_t gpart, lpart, qt, rscale, total;
  };
  int dp() const { return (int)((D + 15) / 16 * 16); }
  int64_t np() const { return (N + kWideRT - 1) / kWideRT * kWideRT; }
  // Chains of a launch: residuals of 1 GB at most, whole chain tiles.
  int64_t lim() const {
    const int64_t l = std::max<int64_t>(kGradCT, ((int64_t)1 << 30) / (4 * N) / kGradCT * kGradCT);
    return std::min<int64_t>(l, (int64_t)sms * kGradCT);
  }
  // [residuals hi, lo | gradient partials | likelihood partials | Q^T | scales of R]
  Layout layout(int64_t chains) const {
    const int64_t cap = std::min(chains, lim());
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    Layout l;
    l.cp = (cap + kWideCT - 1) / kWideCT * kWideCT;
    l.gpart = up(4 * (size_t)N * l.cp);
    l.lpart = l.gpart + up(sizeof(float) * grad_tc_rows(sms, cap, dp()) * (size_t)D);
    l.qt = l.lpart + up(sizeof(double) * (size_t)(np() / kWideRT) * cap);
    l.rscale = l.qt + up(sizeof(float) * (size_t)dp() * l.cp);
    l.total = l.rscale + up(sizeof(float) * (size_t)(np() / 32) * l.cp);
    return l;
  }
};

class LogregWide final : public Target {
 public:
  LogregWide(gbm_context* ctx, int64_t n, int64_t d, float prior_scale)
      : shape_{n, d, ctx->num_sms}, N_(n), D_(d) {
    dim = d;
    dp_ = shape_.dp();
    np_ = shape_.np();
    sms_ = ctx->num_sms;
    err_dev_ = ctx->err_dev;
    inv_var_ = 1.f / (prior_scale * prior_scale);
    log_norm_ = -log((double)prior_scale) - 0.5 * log(2.0 * M_PI);
    lim_ = shape_.lim();
  }

  // False if X or the labels do not fit FP16 pairs, or there is no memory for them.
  bool prepare(gbm_context* ctx, const float* X, const float* y) {
    if (!ym_.try_reserve(sizeof(float) * (size_t)np_) ||
        !y_.try_reserve(sizeof(float) * (size_t)N_) ||
        !xt_.try_reserve(sizeof(float) * (size_t)np_ * dp_))
      return false;
    wide_pack_kernel<<<dim3((unsigned)(np_ / 32), (unsigned)((dp_ + 31) / 32)), dim3(32, 8), 0,
                       ctx->stream>>>(X, y, N_, np_, (int)D_, dp_, xt_.as<float>(),
                                      ym_.as<float>());
    GBM_CUDA(cudaGetLastError());
    GBM_CUDA(cudaMemcpyAsync(y_.ptr, y, sizeof(float) * N_, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    if (!x16_.prepare(ctx, X, ym_.as<float>(), N_, (int)D_, dp_, kGradRT)) return false;
    GBM_CUDA(cudaFuncSetAttribute(wide_products_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem));
    grad_tc_setup<false>();
    return true;
  }

  size_t workspace_bytes(int64_t cap) const override { return shape_.layout(cap).total; }

  void eval(const float* q, int ldq, const int* n_dev, int cap, double* logp, float* grad,
            int ldg, void* ws, cudaStream_t s) override {
    const int N = (int)N_, D = (int)D_, lim = (int)lim_;
    const WideShape::Layout l = shape_.layout(cap);
    char* w = static_cast<char*>(ws);
    __half* rhi = reinterpret_cast<__half*>(w);
    __half* rlo = rhi + (size_t)N_ * l.cp;
    float* gpart = reinterpret_cast<float*>(w + l.gpart);
    double* lpart = reinterpret_cast<double*>(w + l.lpart);
    float* qt = reinterpret_cast<float*>(w + l.qt);
    float* rscale = reinterpret_cast<float*>(w + l.rscale);
    const int rtiles = (int)(np_ / kWideRT), cp = (int)l.cp;
    for (int base = 0; base < cap; base += lim) {
      const int here = std::min(lim, cap - base);
      const float* qc = q + (size_t)base * ldq;
      const int ctiles = (here + kWideCT - 1) / kWideCT;
      wide_states_kernel<<<dim3((unsigned)(ctiles * 2), (unsigned)((dp_ + 31) / 32)), dim3(32, 8),
                           0, s>>>(qc, ldq, n_dev, base, lim, D, dp_, cp, qt);
      wide_products_kernel<<<dim3((unsigned)ctiles, (unsigned)rtiles), kWideThreads, kWideSmem,
                             s>>>(xt_.as<float>(), np_, y_.as<float>(), N, dp_, qt, cp, n_dev,
                                  base, lim, lpart, rhi, rlo, rscale);
      GBM_CUDA(cudaGetLastError());
      const int g = grad_tc_grid(sms_, here, N_, dp_);
      launch_grad_tc<false>(x16_, rhi, rlo, rscale, cp, N, D, dp_, n_dev, base, lim, here, g, gpart,
                            err_dev_, s);
      launch_split_reduce(lpart, gpart, qc, ldq, n_dev, base, lim, here, kGradCT, kGradRT, g, N, D,
                          inv_var_, log_norm_, nullptr, logp + base, grad + (size_t)base * ldg,
                          ldg, s, rtiles);
    }
  }

  int launches_per_eval(int64_t cap) const override {
    return 4 * (int)((cap + lim_ - 1) / lim_);
  }
  double flops(int64_t n) const override { return 4.0 * (double)N_ * D_ * n; }
  double bytes(int64_t n) const override {
    return 4.0 * (double)N_ * D_ + 4.0 * N_ + 8.0 * (double)n * D_ + 8.0 * n;
  }

 private:
  WideShape shape_;
  int64_t N_, D_, np_ = 0, lim_ = 0;
  int dp_ = 16, sms_ = 1;
  float inv_var_ = 1.f;
  double log_norm_ = 0.0;
  int* err_dev_ = nullptr;
  DeviceBuffer xt_, y_, ym_;
  F16Rows x16_;
};

}  // namespace

// grid.y counts row tiles; residuals of a chain tile stay within 2 GB.
static bool wide_holds(int64_t n, int64_t d) {
  constexpr int64_t kMostRows = (int64_t)1 << 22;
  return d > 128 && d <= 256 && n <= kMostRows;
}

std::unique_ptr<Target> make_logreg_wide(gbm_context* ctx, const float* X, int64_t n, int64_t d,
                                         const float* y, float prior_scale) {
  if (!wide_holds(n, d)) return nullptr;
  auto t = std::make_unique<LogregWide>(ctx, n, d, prior_scale);
  if (!t->prepare(ctx, X, y)) return nullptr;
  return t;
}

size_t logreg_wide_bytes(int64_t n, int64_t d, int64_t chains, int num_sms) {
  if (!wide_holds(n, d)) return 0;
  const WideShape w{n, d, num_sms};
  return 4 * (size_t)w.np() * (w.dp() + 1) + 4 * (size_t)n +
         F16Rows::bytes(n, (int)d, w.dp(), num_sms) + w.layout(chains).total;
}

}  // namespace gbm
