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

// Two launches over (chain tiles, output blocks), the blocks with the longest sums
// first.
template <int PHASE, int CT, int OB, int RO, int KG>
struct MvnLaunch {
  static constexpr int kGroups = PHASE == 0 ? 1 : KG;
  static constexpr int kThreads = CT / 4 * (OB / RO) * kGroups;
  using Smem = MvnSmem<CT, OB, kGroups>;
};

template <int PHASE, int CT, int OB, int RO, int KG>
__global__ void __launch_bounds__(MvnLaunch<PHASE, CT, OB, RO, KG>::kThreads)
mvn_tri_kernel(MvnFactor f, const float* __restrict__ A, int lda, const int* __restrict__ n_dev,
               float* __restrict__ out, int ldo, double* __restrict__ part,
               double* __restrict__ logp) {
  using L = MvnLaunch<PHASE, CT, OB, RO, KG>;
  extern __shared__ __align__(16) unsigned char smem[];
  auto& sm = *reinterpret_cast<typename L::Smem*>(smem);
  const int n = *n_dev, c0 = blockIdx.x * CT;
  if (c0 >= n) return;
  const int ob = PHASE == 0 ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  if (threadIdx.x < CT) {
    const int c = c0 + threadIdx.x;
    sm.in[threadIdx.x] = (long long)c * lda;
    sm.out[threadIdx.x] = (long long)c * ldo;
    sm.part[threadIdx.x] = (long long)c * mvn_parts(f.dim);
    sm.id[threadIdx.x] = c;
  }
  mvn_tile<PHASE, CT, OB, 4, RO, L::kGroups>(f, min(CT, n - c0), ob * OB, A, out, part, logp, sm);
}

// The tiles of a target's evaluations, MvnLaunch's parameters.
template <int CT, int OB, int RO, int KG>
struct MvnTiles {
  template <int PHASE>
  static void set_smem() {
    constexpr int bytes = (int)sizeof(typename MvnLaunch<PHASE, CT, OB, RO, KG>::Smem);
    if (bytes > 48 * 1024)    // up to there a launch may ask for it as it is
      GBM_CUDA(cudaFuncSetAttribute(mvn_tri_kernel<PHASE, CT, OB, RO, KG>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  }
  static void prepare() {
    set_smem<0>();
    set_smem<1>();
  }
  template <int PHASE>
  static void launch(const MvnFactor& f, const float* a, int lda, const int* n_dev, int cap,
                     float* out, int ldo, double* part, double* logp, cudaStream_t s) {
    using L = MvnLaunch<PHASE, CT, OB, RO, KG>;
    const dim3 grid((cap + CT - 1) / CT, (f.dim + OB - 1) / OB);
    mvn_tri_kernel<PHASE, CT, OB, RO, KG><<<grid, L::kThreads, sizeof(typename L::Smem), s>>>(
        f, a, lda, n_dev, out, ldo, part, logp);
    GBM_CUDA(cudaGetLastError());
  }
  static void eval(const MvnFactor& f, const float* q, int ldq, const int* n_dev, int cap,
                   float* u, float* grad, int ldg, double* part, double* logp, cudaStream_t s) {
    launch<0>(f, q, ldq, n_dev, cap, u, f.dim, part, logp, s);
    launch<1>(f, u, f.dim, n_dev, cap, grad, ldg, part, logp, s);
  }
};

class Mvn final : public Target {
 public:
  Mvn(gbm_context* ctx, const float* loc, const float* scale_tril_inv, int64_t d,
      double log_norm)
      : sms_(ctx->num_sms) {
    dim = d;
    mu_.reserve(sizeof(float) * d);
    m_.reserve(mvn_factor_bytes(d));
    GBM_CUDA(cudaMemcpyAsync(mu_.ptr, loc, sizeof(float) * d, cudaMemcpyDeviceToDevice,
                             ctx->stream));
    factor_ = mvn_factor(scale_tril_inv, mu_.as<float>(), d, log_norm, m_.as<float>(),
                         ctx->stream);
    for (int64_t chains : {(int64_t)1, kMany * sms_ * 64})
      tiles(chains, [](auto t) { decltype(t)::prepare(); });
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
    tiles(cap, [&](auto t) {
      decltype(t)::eval(factor_, q, ldq, n_dev, cap, u, grad, ldg, part, logp, s);
    });
  }
  int launches_per_eval(int64_t) const override { return 2; }
  // Two triangular GEMMs: ~D^2 multiply-adds each per chain.
  double flops(int64_t n) const override { return 2.0 * (double)dim * dim * n; }
  double bytes(int64_t n) const override {
    return 4.0 * (double)dim * dim + 8.0 * (double)n * dim + 8.0 * n;
  }

 private:
  // The tiles for `chains` chains, passed to `use`.  32 x 64 is the fastest of all
  // tiles up to 2048 x 512 (64 x 64, 4 x 8 a thread: 777 x 350 51 against 56 us before
  // phase 1 was cut, 300 x 2000 41.4 against 38.7).  From kMany tiles an SM on, what
  // counts is the work done, and 64 x 64 does more with a shared load: 1000 x 5000 366
  // us with 32 x 64, 314 so; 65 x 20,000 62 and 50; 1000 x 2000 (under the line) 152
  // and 156.  Vectors of at most 32 have one block of 32 outputs: 2 x 100,000 99 us
  // with 32 x 64, 34 so, and as long as before at any few chains.  Phase 1 cuts k into
  // as many stretches as an output has 32s, at most four: a stretch less is a group
  // of threads less that waits (64 x 20,000 40 us with four, 35 with two), and the
  // sums are the same.
  static constexpr int64_t kMany = 4;
  template <class Use>
  void tiles(int64_t chains, Use&& use) const {
    const bool many = (chains + 63) / 64 * ((dim + 63) / 64) >= kMany * sms_;
    if (dim <= 32)
      use(MvnTiles<64, 32, 4, 1>());
    else if (dim <= 64 && many)
      use(MvnTiles<64, 64, 8, 2>());
    else if (dim <= 64)
      use(MvnTiles<32, 64, 4, 2>());
    else if (many)
      use(MvnTiles<64, 64, 8, 4>());
    else
      use(MvnTiles<32, 64, 4, 4>());
  }

  int sms_ = 1;
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
