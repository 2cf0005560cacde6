// Logistic-regression log-density + gradient above the fused kernels'
// feature limits (FP32 above 256 features, mixed precision above 512): the
// two contractions are plain library GEMMs (cuBLAS, FP32 accumulation) and
// the element-wise work between and after them is this library's own.
//
// Mathematics as in logreg_f32.cu (the inference_gym target,
// spinoffs/inference_gym/inference_gym/targets/logistic_regression.py:92-103,
// distributions/bernoulli.py:126-140):
//   Z = X B^T                       GEMM (N x n), column-major, Z[r + c N]
//   per element: |z|/2 + ln(1 + e^-|z|) summed per chain, R = y - sigmoid(z)
//   G^T = X^T R                     GEMM (D x n) = grad rows [n][D]
//   logp_c = (X^T (y - 1/2)) . q_c - sum_r (|z|/2 + ln(1 + e^-|z|)) + prior
// Mixed precision: X is BF16 (plus a BF16 residual X_lo for FP32 data), the
// states are split into BF16 hi + lo, R into BF16 hi + lo, and the products
// X_hi B_hi^T + X_hi B_lo^T (+ X_lo B_hi^T) and X_hi^T R_hi + X_hi^T R_lo
// (+ X_lo^T R_hi) are accumulated in FP32 -- the residual correction of the
// fused tensor-core kernels.  The hi and lo splits sit side by side as 2n
// columns, so each contraction is one GEMM (plus one for X_lo).  FP32: Z in
// FP32 (no TF32); X^T R from FP16 pairs on the tensor cores (grad_tc.cuh, whose
// partials the split reduction adds), or in FP32 where the data do not fit those.
// 12,289 x 601, 99 chains: 121 us with both GEMMs in FP32, 93 so;
// 60,000 x 1000, 256 chains: 1238 and 718.
//
// This target evaluates all `cap` states of a call (the GEMM shapes are host
// values): a sampler's inactive rows are computed and ignored.  Every GEMM
// and kernel is launched on the call's stream; the cuBLAS workspace is part
// of the target workspace, so evaluations can be captured in CUDA graphs.
#include <cublas_v2.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <string>

#include "engine.h"
#include "grad_tc.cuh"
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr size_t kCublasWs = 32u << 20;   // cuBLAS workspace inside the target workspace
constexpr int kRowBlock = 2048;           // rows per epilogue block
constexpr int kEpiThreads = 64;           // epilogue block: a row block of one chain
constexpr int kEpiRows = kRowBlock / 256;  // rows, 256 apart, of one FP32 sum
constexpr int kEpiBatch = 4;              // of them loaded together
// From kPairRows rows on the FP32 target's X^T R comes from FP16 pairs.  Faster below,
// too (2001 x 300, 64 chains: 61 against 83 us), but there the FP32 GEMM, with few
// additions, is the more exact one (1.5e-7 of the gradient against 1.8e-7).
constexpr float kNegLog2eL = -1.4426950408889634f;
constexpr float kLn2L = 0.6931471805599453f;

#define GBM_CUBLAS(call)                                                          \
  do {                                                                            \
    cublasStatus_t _s = (call);                                                   \
    if (_s != CUBLAS_STATUS_SUCCESS) throw CudaError{cudaErrorUnknown, #call};    \
  } while (0)

// One cuBLAS handle per host thread (and device): creating a handle can
// synchronise, so it happens once, not per target or evaluation.
cublasHandle_t thread_handle(int device) {
  static thread_local cublasHandle_t h[64] = {};
  if (device < 0 || device >= 64) throw CudaError{cudaErrorInvalidDevice, "device index"};
  if (!h[device]) GBM_CUBLAS(cublasCreate(&h[device]));
  return h[device];
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

template <class T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

// What a residual is stored as: its multiple and, for FP16 pairs, the negative
// of the likelihood sums (the split reduction adds, large_finish subtracts).
template <class TO> struct Stored { static constexpr float kScale = 1.f, kSign = 1.f; };
template <> struct Stored<__half> { static constexpr float kScale = kF16Scale, kSign = -1.f; };
template <> __device__ __forceinline__ __half from_float<__half>(float v) {
  return __float2half_rn(v);
}

// X [N][D] (float32 or BF16) -> hi [Np][ld] (and lo for FP32 data in the
// mixed form), zero-padded features; ym = y - 1/2.
// Rows N .. Np - 1 (the padding to a multiple of 8 rows) are zero.
template <class TI, class TO>
__global__ void large_pack_kernel(const TI* __restrict__ X, const float* __restrict__ y,
                                  int64_t N, int64_t Np, int D, int ld, TO* __restrict__ hi,
                                  TO* __restrict__ lo, float* __restrict__ ym) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < Np) ym[i] = i < N ? y[i] - 0.5f : 0.f;
  if (i >= Np * ld) return;
  const int64_t r = i / ld;
  const int d = (int)(i - r * ld);
  const float v = (d < D && r < N) ? (float)X[r * D + d] : 0.f;
  const TO h = from_float<TO>(v);
  hi[i] = h;
  if (lo) lo[i] = from_float<TO>(v - (float)h);
}

// lin[d] = sum_r (y_r - 1/2) X[r][d] in float64, fixed order (two passes).
template <class TI>
__global__ void large_lin_partial(const TI* __restrict__ X, const float* __restrict__ y,
                                  int64_t N, int D, int64_t chunk, double* __restrict__ part) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk;
  const int64_t r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    double acc = 0.0;
    for (int64_t r = r0; r < r1; ++r) acc += ((double)y[r] - 0.5) * (double)(float)X[r * D + d];
    part[(size_t)blockIdx.x * D + d] = acc;
  }
}

__global__ void large_lin_sum(const double* __restrict__ part, int nb, int D,
                              double* __restrict__ lin) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  double acc = 0.0;
  for (int b = 0; b < nb; ++b) acc += part[(size_t)b * D + d];
  lin[d] = acc;
}

// States q [n][ldq] -> B [n][ld] (hi, and lo in the mixed form), zero-padded.
template <class TO>
__global__ void large_split_states(const float* __restrict__ q, int ldq, int n, int D, int ld,
                                   TO* __restrict__ hi, TO* __restrict__ lo) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)n * ld) return;
  const int64_t c = i / ld;
  const int d = (int)(i - c * ld);
  const float v = d < D ? q[c * ldq + d] : 0.f;
  const TO h = from_float<TO>(v);
  hi[i] = h;
  if (lo) lo[i] = from_float<TO>(v - (float)h);
}

// Four consecutive residuals, 8 or 16 bytes.
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <class TO>
__device__ __forceinline__ void store4(TO* p, const float (&v)[4]) {
  TO t[4] = {from_float<TO>(v[0]), from_float<TO>(v[1]), from_float<TO>(v[2]),
             from_float<TO>(v[3])};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(t);
}

// Over Z [n columns][N rows] (column-major): per (row block, chain) the sum
// of |z|/2 + ln(1 + e^-|z|) (float64 partial) and R = (y - 1/2) - sign(z)
// (1/(1 + e^-|z|) - 1/2) (hi, and lo in the mixed form).
//
// What bounds it: memory (in the mixed form Z is as large as the L2 and R half of
// that).  A thread takes four consecutive rows at a time, 16-byte loads, four rows'
// batches in flight; the rows 256 apart that were one thread's when a thread took
// one row stay one FP32 sum.  65,371 rows, 240 chains of hi and lo: 48 us with one
// row a thread, 33 so; blocks of 256 threads and more loads in flight were slower.
template <class TO>
__global__ void __launch_bounds__(kEpiThreads, 16)
large_epilogue(const float* __restrict__ Z, const float* __restrict__ Zlo,
               const float* __restrict__ ym, int64_t N, int64_t ldz, int n,
               TO* __restrict__ Rhi, TO* __restrict__ Rlo, double* __restrict__ part) {
  __shared__ double red;
  const int64_t r0 = (int64_t)blockIdx.x * kRowBlock + 4 * threadIdx.x;
  for (int c = blockIdx.y; c < n; c += gridDim.y) {   // grid.y is capped at 65535
    const size_t col = (size_t)c * ldz;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k0 = 0; k0 < kEpiRows; k0 += kEpiBatch) {
      float4 zv[kEpiBatch], zl[kEpiBatch];
#pragma unroll
      for (int k = 0; k < kEpiBatch; ++k) {
        const int64_t r = r0 + 256 * (k0 + k);
        zv[k] = zl[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < ldz) {      // ldz is a multiple of 8: all four or none
          zv[k] = __ldcs(reinterpret_cast<const float4*>(Z + col + r));
          if (Zlo) zl[k] = __ldcs(reinterpret_cast<const float4*>(Zlo + col + r));
        }
      }
#pragma unroll
      for (int k = 0; k < kEpiBatch; ++k) {
        const int64_t r = r0 + 256 * (k0 + k);
        if (r >= ldz) break;
        const float4 y4 = *reinterpret_cast<const float4*>(ym + r);
        const float yv[4] = {y4.x, y4.y, y4.z, y4.w};
        float z[4] = {zv[k].x, zv[k].y, zv[k].z, zv[k].w};
        if (Zlo) {
          z[0] += zl[k].x;
          z[1] += zl[k].y;
          z[2] += zl[k].z;
          z[3] += zl[k].w;
        }
        float hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          hi[e] = lo[e] = 0.f;     // padding rows: zero residual, no likelihood term
          if (r + e >= N) continue;
          const float a = fabsf(z[e]);
          const float t = tc::ex2_approx(a * kNegLog2eL);
          const float u = 1.f + t;
          acc[e] += fmaf(kLn2L, tc::lg2_approx(u), 0.5f * a);
          const float w = tc::rcp_approx(u) - 0.5f;
          hi[e] = (z[e] >= 0.f ? yv[e] - w : yv[e] + w) * Stored<TO>::kScale;
          lo[e] = hi[e] - (float)from_float<TO>(hi[e]);
        }
        store4(Rhi + col + r, hi);
        if (Rlo) store4(Rlo + col + r, lo);
      }
    }
    const double sum = warp_sum(((double)acc[0] + (double)acc[1]) +
                                ((double)acc[2] + (double)acc[3]));
    if (threadIdx.x == 32) red = sum;
    __syncthreads();
    if (threadIdx.x == 0)
      part[(size_t)blockIdx.x * n + c] = (double)Stored<TO>::kSign * (sum + red);
    __syncthreads();                                   // red of this chain is read
  }
}

// One block per chain: log-density from the partials, the linear term and the
// prior, in a fixed order; gradient G - q / s^2.  (A warp per chain waited for its
// loads in turn: 15 us at 929 features, 240 chains, 8 with 256 threads; from
// kManyChains on, where that leaves the GPU short of chains, 128: 300 x 300, 20,000 of
// them 366 and 328 us an evaluation.)
constexpr int kManyChains = 2048;
template <int kFinishThreads>
__global__ void __launch_bounds__(kFinishThreads)
large_finish(const double* __restrict__ part, int nblk, int n, const float* __restrict__ G,
             const float* __restrict__ Glo, int ld, const float* __restrict__ q, int ldq,
             const double* __restrict__ lin, int D, float inv_var, double log_norm,
             double* __restrict__ logp, float* __restrict__ grad, int ldg) {
  __shared__ double red[kFinishThreads / 32];
  const int c = blockIdx.x, tid = threadIdx.x;
  double t = 0.0;
#pragma unroll 4
  for (int d = tid; d < D; d += kFinishThreads) {
    const float qv = q[(size_t)c * ldq + d];
    t += lin[d] * (double)qv - 0.5 * (double)inv_var * (double)qv * (double)qv;
    const float g = Glo ? G[(size_t)c * ld + d] + Glo[(size_t)c * ld + d] : G[(size_t)c * ld + d];
    grad[(size_t)c * ldg + d] = g - qv * inv_var;
  }
  for (int b = tid; b < nblk; b += kFinishThreads) t -= part[(size_t)b * n + c];
  t = warp_sum(t);
  if ((tid & 31) == 0) red[tid >> 5] = t;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int w = 0; w < kFinishThreads / 32; ++w) s += red[w];
    logp[c] = s + (double)D * log_norm;
  }
}

// Sizes of a target's data and of its workspace.
struct LargeShape {
  int64_t N, D;
  bool mixed;
  int ld() const { return (int)((D + 7) / 8 * 8); }
  // Leading dimension of Z and R: N rounded up to 8 rows.
  int64_t ldz() const { return (N + 7) / 8 * 8; }
  int dp() const { return (int)((D + 15) / 16 * 16); }
  size_t el() const { return mixed ? 2 : 4; }
  // Column sets: the mixed form stacks the hi and lo state (and residual)
  // splits side by side, so each contraction is one GEMM of 2n columns whose
  // halves are added in FP32 by the epilogue (Z) and the finish (G).
  int sets() const { return mixed ? 2 : 1; }
  // tc: X^T R from FP16 pairs.
  size_t g_bytes(int64_t cap, bool tc, int sms) const {
    return tc ? 4 * grad_tc_rows(sms, cap, dp()) * (size_t)D : 4 * (size_t)sets() * cap * ld();
  }
  // [B (sets x n rows) | Z (Np x sets n) | R | G (ld x sets n, or the gradient
  //  partials) | partials | cuBLAS workspace]
  size_t work_bytes(int64_t cap, bool tc, int sms) const {
    const size_t w = (size_t)sets() * cap, nblk = (size_t)((N + kRowBlock - 1) / kRowBlock);
    return align256(el() * w * ld()) + align256(4 * (size_t)ldz() * w) +
           align256(el() * (size_t)ldz() * w) + align256(g_bytes(cap, tc, sms)) +
           align256(8 * nblk * cap) + kCublasWs;
  }
};

class LogregLarge final : public Target {
 public:
  LogregLarge(gbm_context* ctx, const void* X, int x_dtype, int64_t n, int64_t d, const float* y,
              float prior_scale, bool mixed, bool pairs)
      : shape_{n, d, mixed}, N_(n), D_(d), mixed_(mixed), device_(ctx->device) {
    dim = d;
    ld_ = shape_.ld();
    ldz_ = shape_.ldz();
    xlo_ = mixed && x_dtype == 0;
    const size_t el = shape_.el();
    xh_.reserve(el * (size_t)ldz_ * ld_);
    if (xlo_) xl_.reserve(el * (size_t)ldz_ * ld_);
    ym_.reserve(sizeof(float) * (size_t)ldz_);
    const int64_t total = ldz_ * ld_;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    cudaStream_t s = ctx->stream;
    if (mixed && x_dtype == 0)
      large_pack_kernel<float, __nv_bfloat16><<<blocks, 256, 0, s>>>(
          static_cast<const float*>(X), y, N_, ldz_, (int)D_, ld_, xh_.as<__nv_bfloat16>(),
          xl_.as<__nv_bfloat16>(), ym_.as<float>());
    else if (mixed)
      large_pack_kernel<__nv_bfloat16, __nv_bfloat16><<<blocks, 256, 0, s>>>(
          static_cast<const __nv_bfloat16*>(X), y, N_, ldz_, (int)D_, ld_,
          xh_.as<__nv_bfloat16>(), nullptr, ym_.as<float>());
    else
      large_pack_kernel<float, float><<<blocks, 256, 0, s>>>(
          static_cast<const float*>(X), y, N_, ldz_, (int)D_, ld_, xh_.as<float>(), nullptr,
          ym_.as<float>());
    GBM_CUDA(cudaGetLastError());
    {
      const int nb = 2 * ctx->num_sms;
      const int64_t chunk = (N_ + nb - 1) / nb;
      DeviceBuffer part;
      part.reserve(sizeof(double) * (size_t)nb * D_);
      lin_.reserve(sizeof(double) * (size_t)D_);
      if (x_dtype == 0)
        large_lin_partial<<<nb, 256, 0, s>>>(static_cast<const float*>(X), y, N_, (int)D_, chunk,
                                             part.as<double>());
      else
        large_lin_partial<<<nb, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(X), y, N_,
                                             (int)D_, chunk, part.as<double>());
      large_lin_sum<<<(unsigned)((D_ + 127) / 128), 128, 0, s>>>(part.as<double>(), nb,
                                                                 (int)D_, lin_.as<double>());
      GBM_CUDA(cudaGetLastError());
      GBM_CUDA(cudaStreamSynchronize(s));   // `part` is freed on scope exit
    }
    sms_ = ctx->num_sms;
    err_dev_ = ctx->err_dev;
    dp_ = shape_.dp();
    tc_ = pairs && !mixed && n >= kPairRows &&
          x16_.prepare(ctx, static_cast<const float*>(X), ym_.as<float>(), N_, (int)D_, dp_,
                       kGradRT);
    if (tc_) grad_tc_setup<true>();
    inv_var_ = 1.f / (prior_scale * prior_scale);
    log_norm_ = -log((double)prior_scale) - 0.5 * log(2.0 * M_PI);
  }

  size_t workspace_bytes(int64_t cap) const override {
    return shape_.work_bytes(cap, tc_, sms_);
  }

  void eval(const float* q, int ldq, const int*, int cap, double* logp, float* grad, int ldg,
            void* ws, cudaStream_t s) override {
    const size_t el = mixed_ ? 2 : 4;
    const int64_t nblk = (N_ + kRowBlock - 1) / kRowBlock;
    const int n = cap, w = shape_.sets() * cap, D = (int)D_;
    unsigned char* p = static_cast<unsigned char*>(ws);
    unsigned char* B = p;          p += align256(el * (size_t)w * ld_);
    float* Z = reinterpret_cast<float*>(p);    p += align256(4 * (size_t)ldz_ * w);
    unsigned char* R = p;          p += align256(el * (size_t)ldz_ * w);
    float* G = reinterpret_cast<float*>(p);    p += align256(shape_.g_bytes(cap, tc_, sms_));
    double* part = reinterpret_cast<double*>(p); p += align256(8 * (size_t)nblk * cap);
    void* cws = p;
    cublasHandle_t h = thread_handle(device_);
    GBM_CUBLAS(cublasSetStream(h, s));
    GBM_CUBLAS(cublasSetWorkspace(h, cws, kCublasWs));
    const unsigned sb = (unsigned)(((int64_t)n * ld_ + 255) / 256);
    if (mixed_)
      large_split_states<__nv_bfloat16><<<sb, 256, 0, s>>>(
          q, ldq, n, D, ld_, reinterpret_cast<__nv_bfloat16*>(B),
          reinterpret_cast<__nv_bfloat16*>(B) + (size_t)n * ld_);
    else
      large_split_states<float><<<sb, 256, 0, s>>>(q, ldq, n, D, ld_,
                                                   reinterpret_cast<float*>(B), nullptr);
    GBM_CUDA(cudaGetLastError());
    const cudaDataType_t dt = mixed_ ? CUDA_R_16BF : CUDA_R_32F;
    const float one = 1.f, zero = 0.f;
    // Z = X_hi [B_hi; B_lo]^T (+ X_lo B_hi^T into the first n columns):
    // column-major (Np x w) over the rows padded to a multiple of 8 and the
    // ld_ zero-padded features: every extent the GEMMs see is a multiple of 8
    // elements, so the library picks its aligned tensor-core kernels (with an
    // odd row count it falls back to element-aligned ones, ~15x slower here);
    // the padding of X and of B is zero, so the sums are unchanged.
    const int Kp = ld_, ldz = (int)ldz_;
    auto gemm_z = [&](const void* xa, int cols, const float* beta) {
      GBM_CUBLAS(cublasGemmEx(h, CUBLAS_OP_T, CUBLAS_OP_N, ldz, cols, Kp, &one, xa, dt, ld_, B,
                              dt, ld_, beta, Z, CUDA_R_32F, ldz, CUBLAS_COMPUTE_32F,
                              CUBLAS_GEMM_DEFAULT));
    };
    gemm_z(xh_.ptr, w, &zero);
    if (xlo_) gemm_z(xl_.ptr, n, &one);
    const float* Zlo = mixed_ ? Z + (size_t)n * ldz_ : nullptr;
    const dim3 eg((unsigned)nblk, (unsigned)std::min(n, 65535));
    if (mixed_)
      large_epilogue<__nv_bfloat16><<<eg, kEpiThreads, 0, s>>>(
          Z, Zlo, ym_.as<float>(), N_, ldz_, n, reinterpret_cast<__nv_bfloat16*>(R),
          reinterpret_cast<__nv_bfloat16*>(R) + (size_t)n * ldz_, part);
    else if (tc_)
      large_epilogue<__half><<<eg, kEpiThreads, 0, s>>>(Z, nullptr, ym_.as<float>(), N_, ldz_, n,
                                                reinterpret_cast<__half*>(R),
                                                reinterpret_cast<__half*>(R) + (size_t)n * ldz_,
                                                part);
    else
      large_epilogue<float><<<eg, kEpiThreads, 0, s>>>(Z, nullptr, ym_.as<float>(), N_, ldz_, n,
                                               reinterpret_cast<float*>(R), nullptr, part);
    GBM_CUDA(cudaGetLastError());
    if (tc_) {
      __half* r = reinterpret_cast<__half*>(R);
      const int g = grad_tc_grid(sms_, n, N_, dp_);
      launch_grad_tc<true>(x16_, r, r + (size_t)n * ldz_, nullptr, ldz_, (int)N_, D, dp_,
                           nullptr, 0, n, n, g, G, err_dev_, s);
      launch_split_reduce(part, G, q, ldq, nullptr, 0, n, n, kGradCT, kGradRT, g, (int)N_, D,
                          inv_var_, log_norm_, lin_.as<double>(), logp, grad, ldg, s, (int)nblk);
      return;
    }
    // G^T = X_hi^T [R_hi | R_lo] (+ X_lo^T R_hi into the first n columns):
    // column-major (ld x w) over all ld_ padded features (rows >= D come out
    // zero and are not read) and the Np padded rows (zero residuals).
    auto gemm_g = [&](const void* xa, int cols, const float* beta) {
      GBM_CUBLAS(cublasGemmEx(h, CUBLAS_OP_N, CUBLAS_OP_N, Kp, cols, ldz, &one, xa, dt, ld_, R,
                              dt, ldz, beta, G, CUDA_R_32F, ld_, CUBLAS_COMPUTE_32F,
                              CUBLAS_GEMM_DEFAULT));
    };
    gemm_g(xh_.ptr, w, &zero);
    if (xlo_) gemm_g(xl_.ptr, n, &one);
    auto finish = [&](auto kernel, int threads) {
      kernel<<<(unsigned)n, threads, 0, s>>>(part, (int)nblk, n, G,
                                             mixed_ ? G + (size_t)n * ld_ : nullptr, ld_, q, ldq,
                                             lin_.as<double>(), D, inv_var_, log_norm_, logp, grad,
                                             ldg);
    };
    if (n >= kManyChains)
      finish(large_finish<128>, 128);
    else
      finish(large_finish<256>, 256);
    GBM_CUDA(cudaGetLastError());
  }

  // split, epilogue, finish (or gradient and reduction) + the GEMMs (library
  // kernels, not counted).
  int launches_per_eval(int64_t) const override { return tc_ ? 4 : 3; }
  double flops(int64_t n) const override { return 4.0 * (double)N_ * D_ * n; }
  double bytes(int64_t n) const override {
    return (mixed_ ? 2.0 : 4.0) * (double)N_ * D_ + 4.0 * N_ + 8.0 * (double)n * D_ + 8.0 * n;
  }

 private:
  LargeShape shape_;
  int64_t N_, D_;
  bool tc_ = false;              // X^T R from FP16 pairs
  int sms_ = 1, dp_ = 16;
  int* err_dev_ = nullptr;
  F16Rows x16_;
  bool mixed_, xlo_ = false;
  int device_ = 0, ld_ = 8;
  int64_t ldz_ = 8;
  float inv_var_ = 1.f;
  double log_norm_ = 0.0;
  DeviceBuffer xh_, xl_, ym_, lin_;
};

}  // namespace

std::unique_ptr<Target> make_logreg_large(gbm_context* ctx, const void* X, int x_dtype, int64_t n,
                                          int64_t d, const float* y, float prior_scale,
                                          bool mixed, bool pairs) {
  if (n >= ((int64_t)1 << 31) || d >= ((int64_t)1 << 20)) return nullptr;   // GEMM dimensions
  return std::unique_ptr<Target>(
      new LogregLarge(ctx, X, x_dtype, n, d, y, prior_scale, mixed, pairs));
}

size_t logreg_large_bytes(int64_t n, int64_t d, int64_t chains, int num_sms, bool mixed,
                          int x_dtype, bool pairs) {
  const LargeShape h{n, d, mixed};
  const bool tc = pairs && !mixed && n >= kPairRows;
  const size_t x = h.el() * (size_t)h.ldz() * h.ld();
  return x * (mixed && x_dtype == 0 ? 2 : 1) + 4 * (size_t)h.ldz() +
         8 * (size_t)d * (2 * num_sms + 1) +
         (tc ? F16Rows::bytes(n, (int)d, h.dp(), num_sms) : 0) +
         std::max(h.work_bytes(chains, tc, num_sms), h.work_bytes(chains, false, num_sms));
}

}  // namespace gbm
