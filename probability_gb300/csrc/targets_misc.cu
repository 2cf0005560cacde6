// Multivariate-normal and non-centred hierarchical-normal targets.
//
// MultivariateNormalTriL (distributions/mvn_tril.py:44, log_prob through
// mvn_linear_operator.py:242, which solves with the scale factor L):
//   u = L^-1 (x - mu),  logp = -1/2 |u|^2 + log_norm,  grad = -L^-T u
// with L^-1 and log_norm = -sum log|L_ii| - D/2 log 2pi supplied by the
// caller (computed once from scale_tril).  Working with L^-1 keeps the
// conditioning of L (the square root of the covariance's) -- multiplying by
// the precision L^-T L^-1 in FP32 would square it.  Both products are
// triangular GEMMs over all chains on the CUDA cores (mvn_tile.cuh), one launch
// each; the first also forms sums of u^2 over 32 outputs, which the second adds
// in fixed order (deterministic).
//
// Non-centred hierarchical normal, the eight-schools pattern of
// mcmc/eight_schools_hmc.py:41-58 with mu ~ N(0, s_mu), tau ~ HalfCauchy(0,
// s_tau) (distributions/half_cauchy.py:138-145) sampled as log tau with its
// log-Jacobian, z_j ~ N(0, 1), y_j ~ N(mu + tau z_j, sigma_j).  State =
// [mu, log tau, z_1..z_J]; one warp per chain.
#include <cuda_runtime.h>

#include <memory>

#include "engine.h"
#include "mvn_tile.cuh"
#include "nuts_chain.h"

namespace gbm {
namespace {

// Two launches over (chain tiles, output blocks), the blocks with the longest
// sums first.  The tile is 32 x 64 at every size: 32 x 32 and 64 x 64 (4 x 8 a
// thread) tiles were slower from 8 x 32 chains to 2048 x 512 (777 x 350, before
// phase 1 was cut: 56, 51 and 83 us), and four groups halve phase 1.
constexpr int kMvnCT = 32, kMvnOB = 64;

template <int PHASE>
struct MvnLaunch {
  static constexpr int kGroups = PHASE == 0 ? 1 : 4;
  static constexpr int kThreads = kMvnCT / 4 * (kMvnOB / 4) * kGroups;
  using Smem = MvnSmem<kMvnCT, kMvnOB, kGroups>;
};

template <int PHASE>
__global__ void __launch_bounds__(MvnLaunch<PHASE>::kThreads)
mvn_tri_kernel(MvnFactor f, const float* __restrict__ A, int lda, const int* __restrict__ n_dev,
               float* __restrict__ out, int ldo, double* __restrict__ part,
               double* __restrict__ logp) {
  extern __shared__ __align__(16) unsigned char smem[];
  auto& sm = *reinterpret_cast<typename MvnLaunch<PHASE>::Smem*>(smem);
  const int n = *n_dev, c0 = blockIdx.x * kMvnCT;
  if (c0 >= n) return;
  const int ob = PHASE == 0 ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  if (threadIdx.x < kMvnCT) {
    const int c = c0 + threadIdx.x;
    sm.in[threadIdx.x] = (long long)c * lda;
    sm.out[threadIdx.x] = (long long)c * ldo;
    sm.part[threadIdx.x] = (long long)c * mvn_parts(f.dim);
    sm.id[threadIdx.x] = c;
  }
  mvn_tile<PHASE, kMvnCT, kMvnOB, 4, 4, MvnLaunch<PHASE>::kGroups>(
      f, min(kMvnCT, n - c0), ob * kMvnOB, A, out, part, logp, sm);
}

class Mvn final : public Target {
 public:
  Mvn(gbm_context* ctx, const float* loc, const float* scale_tril_inv, int64_t d,
      double log_norm) {
    dim = d;
    mu_.reserve(sizeof(float) * d);
    m_.reserve(mvn_factor_bytes(d));
    GBM_CUDA(cudaMemcpyAsync(mu_.ptr, loc, sizeof(float) * d, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    factor_ = mvn_factor(scale_tril_inv, mu_.as<float>(), d, log_norm, m_.as<float>(),
                         ctx->stream);
    GBM_CUDA(cudaFuncSetAttribute(mvn_tri_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(MvnLaunch<0>::Smem)));
    GBM_CUDA(cudaFuncSetAttribute(mvn_tri_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(MvnLaunch<1>::Smem)));
  }
  static size_t work_bytes(int64_t cap, int64_t d) {
    return sizeof(double) * (size_t)cap * mvn_parts(d) + sizeof(float) * (size_t)cap * d + 512;
  }
  size_t workspace_bytes(int64_t cap) const override { return work_bytes(cap, dim); }
  void eval(const float* q, int ldq, const int* n_dev, int cap, double* logp, float* grad,
            int ldg, void* ws, cudaStream_t s) override {
    double* part = static_cast<double*>(ws);
    float* u = reinterpret_cast<float*>(part + (size_t)cap * mvn_parts(dim));
    const int D = (int)dim;
    const dim3 grid((cap + kMvnCT - 1) / kMvnCT, (D + kMvnOB - 1) / kMvnOB);
    mvn_tri_kernel<0><<<grid, MvnLaunch<0>::kThreads, sizeof(MvnLaunch<0>::Smem), s>>>(
        factor_, q, ldq, n_dev, u, D, part, logp);
    mvn_tri_kernel<1><<<grid, MvnLaunch<1>::kThreads, sizeof(MvnLaunch<1>::Smem), s>>>(
        factor_, u, D, n_dev, grad, ldg, part, logp);
    GBM_CUDA(cudaGetLastError());
  }
  int launches_per_eval(int64_t) const override { return 2; }
  // Two triangular GEMMs: ~D^2 multiply-adds each per chain.
  double flops(int64_t n) const override { return 2.0 * (double)dim * dim * n; }
  double bytes(int64_t n) const override {
    return 4.0 * (double)dim * dim + 8.0 * (double)n * dim + 8.0 * n;
  }

 private:
  MvnFactor factor_{};
  DeviceBuffer mu_, m_;
};

// ---------------------------------------------------------------------------
__global__ void hier_kernel(const float* __restrict__ Q, int ldq, const int* __restrict__ n_dev,
                            int J, const float* __restrict__ y, const float* __restrict__ sigma,
                            float mu_scale, float tau_scale, double const_term,
                            double* __restrict__ logp, float* __restrict__ G, int ldg) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= *n_dev) return;
  const float* x = Q + (size_t)c * ldq;
  const float mu = x[0], eta = x[1];
  const float tau = expf(eta);
  float lp = 0.f, gmu = 0.f, geta = 0.f;
  for (int j = lane; j < J; j += 32) {
    const float z = x[2 + j];
    const float s = sigma[j];
    const float res = (y[j] - (mu + tau * z)) / s;    // standardized residual
    const float r = res / s;                           // d/dtheta log N(y; theta, s)
    lp += -0.5f * z * z - 0.5f * res * res;
    gmu += r;
    geta += r * z;
    G[(size_t)c * ldg + 2 + j] = -z + tau * r;
  }
  double lpd = warp_sum((double)lp);
  gmu = warp_sum(gmu);
  geta = warp_sum(geta);
  if (lane == 0) {
    const float t = tau / tau_scale;
    // priors: mu ~ N(0, s_mu); tau ~ HalfCauchy(0, s_tau) with log-Jacobian eta
    lpd += -0.5 * (double)(mu / mu_scale) * (double)(mu / mu_scale) - log1p((double)t * t) +
           (double)eta + const_term;
    logp[c] = lpd;
    G[(size_t)c * ldg + 0] = -mu / (mu_scale * mu_scale) + gmu;
    G[(size_t)c * ldg + 1] = -2.f * t * t / (1.f + t * t) + 1.f + tau * geta;
  }
}

class Hier final : public Target {
 public:
  Hier(gbm_context* ctx, const float* y, const float* sigma, int64_t J, float mu_scale,
       float tau_scale, double const_term)
      : J_(J), mu_scale_(mu_scale), tau_scale_(tau_scale), const_(const_term) {
    dim = J + 2;
    y_.reserve(sizeof(float) * J);
    s_.reserve(sizeof(float) * J);
    GBM_CUDA(cudaMemcpyAsync(y_.ptr, y, sizeof(float) * J, cudaMemcpyDeviceToDevice, ctx->stream));
    GBM_CUDA(cudaMemcpyAsync(s_.ptr, sigma, sizeof(float) * J, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    if (dim <= kChainMaxDim) {
      const std::vector<double> table = chain_log_table();
      table_.reserve(sizeof(double) * table.size());
      GBM_CUDA(cudaMemcpyAsync(table_.ptr, table.data(), sizeof(double) * table.size(),
                               cudaMemcpyHostToDevice, ctx->stream));
      const HierModel m{y_.as<float>(), s_.as<float>(), mu_scale,
                        tau_scale,      const_term,     table_.as<double>()};
      model_.reserve(sizeof(m));
      GBM_CUDA(cudaMemcpyAsync(model_.ptr, &m, sizeof(m), cudaMemcpyHostToDevice, ctx->stream));
      GBM_CUDA(cudaStreamSynchronize(ctx->stream));   // m, table are this call's
      chain_models_ = ChainModels{model_.as<HierModel>(), nullptr, (int)dim, true};
    }
  }
  size_t workspace_bytes(int64_t) const override { return 256; }
  const ChainModels* chain_models() const override {
    return model_.ptr ? &chain_models_ : nullptr;
  }
  void eval(const float* q, int ldq, const int* n_dev, int cap, double* logp, float* grad,
            int ldg, void*, cudaStream_t s) override {
    hier_kernel<<<(cap + 7) / 8, 256, 0, s>>>(q, ldq, n_dev, (int)J_, y_.as<float>(),
                                              s_.as<float>(), mu_scale_, tau_scale_, const_,
                                              logp, grad, ldg);
    GBM_CUDA(cudaGetLastError());
  }
  int launches_per_eval(int64_t) const override { return 1; }
  double flops(int64_t n) const override { return 10.0 * (double)J_ * n; }
  double bytes(int64_t n) const override { return 8.0 * J_ + 8.0 * (double)(J_ + 2) * n + 8.0 * n; }

 private:
  int64_t J_;
  float mu_scale_, tau_scale_;
  double const_;
  DeviceBuffer y_, s_, model_, table_;
  ChainModels chain_models_{};
};

}  // namespace

size_t mvn_bytes(int64_t d, int64_t chains) {
  return sizeof(float) * (size_t)d + mvn_factor_bytes(d) + Mvn::work_bytes(chains, d);
}

size_t hier_bytes(int64_t groups) {
  return 2 * sizeof(float) * (size_t)groups + sizeof(double) * chain_log_table().size() +
         sizeof(HierModel) + 256;
}

std::unique_ptr<Target> make_mvn(gbm_context* ctx, const float* loc, const float* scale_tril_inv,
                                 int64_t d, double log_norm) {
  return std::unique_ptr<Target>(new Mvn(ctx, loc, scale_tril_inv, d, log_norm));
}

std::unique_ptr<Target> make_hier(gbm_context* ctx, const float* y, const float* sigma, int64_t J,
                                  float mu_scale, float tau_scale) {
  // Constant part of the log-density: HalfCauchy and Normal normalizers.
  std::unique_ptr<float[]> hs(new float[J]);
  GBM_CUDA(cudaMemcpyAsync(hs.get(), sigma, sizeof(float) * J, cudaMemcpyDeviceToHost,
                           ctx->stream));
  GBM_CUDA(cudaStreamSynchronize(ctx->stream));
  const double log2pi = log(2.0 * M_PI);
  double c = log(2.0 / M_PI) - log((double)mu_scale) - log((double)tau_scale) -
             0.5 * (1.0 + 2.0 * (double)J) * log2pi;
  for (int64_t j = 0; j < J; ++j) c -= log((double)hs[j]);
  return std::unique_ptr<Target>(new Hier(ctx, y, sigma, J, mu_scale, tau_scale, c));
}

}  // namespace gbm
