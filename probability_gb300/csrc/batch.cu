// Many independent posteriors of uneven dimension in one NUTS sampler.
//
// The members are multivariate normals (MultivariateNormalTriL,
// distributions/mvn_tril.py:44, with the arithmetic of targets_misc.cu) and
// non-centred hierarchical normals (the eight-schools pattern of
// mcmc/eight_schools_hmc.py:41-58).  Their chains are concatenated into one
// ragged population: member t owns chains [c_begin, c_end), and chain c's
// state vector has dim(t) elements at element offset coff[c].  The NUTS
// kernels run on the whole population at once (per-chain step sizes, one
// launch per sampler step for all members), so a leaf of the sampler costs a
// fixed number of launches however many posteriors are in flight.
//
// Gradient evaluation of the active chains is two persistent launches over
// tile lists built on the device each leaf:
//   schedule: for each member, its active chains are a contiguous run of the
//             (sorted) active list; MVN members contribute
//             ceil(active / ct) x ceil(D / 64) tiles, hierarchical members
//             ceil(active / 4) (more chains a tile where there are very many),
//             those with the longest sums first.
//   phase 0:  MVN tiles form u = L^-1 (x - loc) for a block of 64 rows of u
//             and its |u|^2; hierarchical tiles do all their work.
//   phase 1:  MVN tiles form grad = -L^-T u for a block of 64 columns; the
//             last column block's tile also adds the |u|^2 sums (fixed order).
// CTAs take tiles from the list as they get done, so large and small members
// share the machine in one launch.  The chain-tile width ct (32 or 64 chains) is
// chosen per size class of D by timing both at construction (the autotuner).
//
// What bounds it: mvn_tile.cuh's tiles, and their longest sum where one large
// member holds most of the work.  Twelve normals up to 2048 (497 chains) and
// twelve hierarchical members: 521 us an evaluation with tiles of 128 outputs in
// member order at a fixed stride, 207 now; members of at most 300: 66 and 41.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "engine.h"
#include "gb300_mcmc.h"
#include "mvn_tile.cuh"
#include "nuts_chain.h"

namespace gbm {
namespace {

enum BatchFamily : int { kBatchMvn = 1, kBatchHier = 2 };   // the GBM_FAMILY_* values

constexpr int kOB = 64;          // rows / columns of u or grad per MVN tile
constexpr int kThreads = 128;
// Chains of a hierarchical tile, a multiple of its four warps: four, and up to 32 of
// short vectors where the batch's hierarchical chains still make 16 tiles for each
// SM and more (taking a tile costs about as much as a short chain, and the warps of
// one wait for each other): 2^20 chains of two groups 2750 us an evaluation with four,
// 2330 so; 65,536 of 100 groups 214 and 187.  With 32 tiles an SM as the line 195, with
// 4 196; vectors of 500 are slower with more than four (16,384 chains 87 and 91).
inline int hier_tile_chains(int64_t all_chains, int dim, int num_sms) {
  int ct = 4;
  while (ct < 32 && (int64_t)2 * ct * dim <= 2048 &&
         all_chains >= (int64_t)2 * ct * 16 * num_sms)
    ct *= 2;
  return ct;
}
constexpr int kClasses = 4;      // size classes of D for the tile autotuner

__host__ __device__ inline int size_class(int d) {
  return d <= 64 ? 0 : d <= 256 ? 1 : d <= 1024 ? 2 : 3;
}

struct BDesc {
  int family, dim, c_begin, c_end;
  long long p_begin;    // first |u|^2 partial of this member
  int ct;               // chain tile
  MvnFactor mvn;
  const float* y;
  const float* sigma;
  float mu_scale, tau_scale;
  double hconst;
};

__device__ __forceinline__ int lower_bound_dev(const int* a, int n, int v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (a[m] < v) lo = m + 1; else hi = m;
  }
  return lo;
}

// What a tile of the list works on: `group` of a phase's order, its k-th run of
// chains.
struct Group {
  int member, ob;       // output block (MVN)
};

// Exclusive prefix sum over the block (1024 threads); the total in *total.
__device__ int block_prefix(int v, int* total) {
  __shared__ int warps[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(~0u, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();   // the last call's readers are done
  if (lane == 31) warps[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = warps[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(~0u, w, o);
      if (lane >= o) w += y;
    }
    warps[lane] = w;
  }
  __syncthreads();
  *total = warps[31];
  return x - v + (warp > 0 ? warps[warp - 1] : 0);
}

// Blocks (p, *) write phase p's tile list: {group, run of chains} of every tile in
// the order of the groups; block (p, 0) also their number and the counter that the
// phase takes tiles from, block (0, 0) each member's run [a, a + na) of the active
// list.  Groups may have any number of tiles (a member of 2^20 chains: 2^18), so the
// tiles and not the groups are shared out among the threads, each of which looks up
// its tile's group, and among as many blocks as make about 8 tiles a thread.  2^20
// chains of one member (two groups): 5200 us an evaluation with a group's tiles
// written by one thread, 2750 so, 2330 with larger tiles (hier_tile_chains); 65,536
// chains 352, 202 and 175.
__global__ void __launch_bounds__(1024)
batch_schedule_kernel(const BDesc* __restrict__ d, int T, const int* __restrict__ act,
                      const int* __restrict__ act_count, const Group* __restrict__ groups0,
                      const Group* __restrict__ groups1, int n0, int n1, int* __restrict__ a,
                      int* __restrict__ na, int2* __restrict__ tiles0, int2* __restrict__ tiles1,
                      int* __restrict__ totals, int* __restrict__ next) {
  __shared__ int first[1024];        // tile of the batch of groups that is its group's first
  const int n = *act_count, phase = blockIdx.x;
  const bool lead = blockIdx.y == 0;
  const Group* groups = phase == 0 ? groups0 : groups1;
  int2* tiles = phase == 0 ? tiles0 : tiles1;
  const int ng = phase == 0 ? n0 : n1;
  if (phase == 0 && lead)
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
      const int lo = lower_bound_dev(act, n, d[t].c_begin);
      a[t] = lo;
      na[t] = lower_bound_dev(act, n, d[t].c_end) - lo;
    }
  int done = 0;
  for (int g0 = 0; g0 < ng; g0 += 1024) {
    const int g = g0 + threadIdx.x;
    int runs = 0;
    if (g < ng) {
      const BDesc& m = d[groups[g].member];
      const int ct = m.ct;
      const int held = lower_bound_dev(act, n, m.c_end) - lower_bound_dev(act, n, m.c_begin);
      runs = (held + ct - 1) / ct;
    }
    int total;
    first[threadIdx.x] = block_prefix(runs, &total);
    __syncthreads();
    for (int i = blockIdx.y * 1024 + threadIdx.x; i < total; i += gridDim.y * 1024) {
      int lo = 0;                    // the last group whose first tile is not past i
#pragma unroll
      for (int step = 512; step > 0; step >>= 1)
        if (first[lo + step] <= i) lo += step;
      tiles[done + i] = make_int2(g0 + lo, i - first[lo]);
    }
    __syncthreads();
    done += total;
  }
  if (threadIdx.x == 0 && lead) {
    totals[phase] = done;
    next[phase] = 0;
  }
}

// One hierarchical tile: a warp per chain (targets_misc.cu hier_kernel), every fourth
// of the tile's chains.
__device__ void hier_tile(const BDesc& d, const int* __restrict__ act, int a0, int nc,
                          const int64_t* __restrict__ coff, const float* __restrict__ Q,
                          double* __restrict__ logp, float* __restrict__ Gout) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = w; i < nc; i += kThreads / 32) {
    const int c = act[a0 + i];
    const float* x = Q + coff[c];
    float* G = Gout + coff[c];
    const int J = d.dim - 2;
    const float mu = x[0], eta = x[1];
    const float tau = expf(eta);
    float lp = 0.f, gmu = 0.f, geta = 0.f;
    // Four groups per lane per pass: their loads are issued before any use, so
    // a pass waits for memory once instead of four times.
    for (int j0 = lane; j0 < J; j0 += 128) {
      float z[4], sg[4], yy[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + 32 * u;
        z[u] = j < J ? x[2 + j] : 0.f;
        sg[u] = j < J ? d.sigma[j] : 1.f;
        yy[u] = j < J ? d.y[j] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + 32 * u;
        if (j >= J) break;
        const float res = (yy[u] - (mu + tau * z[u])) / sg[u];
        const float r = res / sg[u];
        lp += -0.5f * z[u] * z[u] - 0.5f * res * res;
        gmu += r;
        geta += r * z[u];
        G[2 + j] = -z[u] + tau * r;
      }
    }
    double lpd = warp_sum((double)lp);
    gmu = warp_sum(gmu);
    geta = warp_sum(geta);
    if (lane == 0) {
      const float t = tau / d.tau_scale;
      lpd += -0.5 * (double)(mu / d.mu_scale) * (double)(mu / d.mu_scale) - log1p((double)t * t) +
             (double)eta + d.hconst;
      logp[c] = lpd;
      G[0] = -mu / (d.mu_scale * d.mu_scale) + gmu;
      G[1] = -2.f * t * t / (1.f + t * t) + 1.f + tau * geta;
    }
  }
}

// A phase's CTAs: phase 0 in groups of 128 threads, as many as fit an SM; phase 1
// with four such groups a CTA, which share the k of a tile.
template <int PHASE>
struct PhaseLaunch {
  static constexpr int kGroups = PHASE == 0 ? 1 : 4;
  static constexpr int kSmem =
      (int)std::max(sizeof(MvnSmem<64, kOB, kGroups>), sizeof(MvnSmem<32, kOB, kGroups>));
};

template <int PHASE, int CT, int RO>
__device__ void run_mvn(const BDesc& d, int o0, const int* __restrict__ act, int a0, int nc,
                        const int64_t* __restrict__ coff, const float* __restrict__ X,
                        float* __restrict__ out, double* __restrict__ part,
                        double* __restrict__ logp, unsigned char* smem) {
  constexpr int KG = PhaseLaunch<PHASE>::kGroups;
  auto& sm = *reinterpret_cast<MvnSmem<CT, kOB, KG>*>(smem);
  if (threadIdx.x < CT) {
    const int i = threadIdx.x, c = i < nc ? act[a0 + i] : d.c_begin;
    sm.id[i] = c;
    sm.in[i] = sm.out[i] = coff[c];
    sm.part[i] = d.p_begin + (long long)(c - d.c_begin) * mvn_parts(d.dim);
  }
  mvn_tile<PHASE, CT, kOB, 4, RO, KG>(d.mvn, nc, o0, X, out, part, logp, sm);
}

// Persistent CTAs.  The list begins with the longest tiles.  A CTA's first tile
// is its place in it, every second stretch of the GPU's SMs counting backwards, so
// that the CTAs that share an SM (as they are placed on an idle GPU: b, b + SMs,
// ...) get about the same work in sum; then each takes the next one left.
template <int PHASE>
__global__ void __launch_bounds__(kThreads * PhaseLaunch<PHASE>::kGroups, PHASE == 0 ? 4 : 1)
batch_phase_kernel(const BDesc* __restrict__ desc, const Group* __restrict__ groups,
                   const int2* __restrict__ tiles, const int* __restrict__ total_dev,
                   int* __restrict__ next, int sms, const int* __restrict__ act,
                   const int* __restrict__ a, const int* __restrict__ na,
                   const int64_t* __restrict__ coff, const float* __restrict__ q,
                   float* __restrict__ u, float* __restrict__ grad, double* __restrict__ part,
                   double* __restrict__ logp) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int taken[2];   // the next tile, of even and odd turns
  const int total = *total_dev, stretch = blockIdx.x / sms, place = blockIdx.x % sms;
  int tile = stretch * sms + (stretch & 1 ? sms - 1 - place : place);
  for (int turn = 0; tile < total; turn ^= 1) {
    const int2 at = tiles[tile];
    const Group g = groups[at.x];
    const BDesc& d = desc[g.member];
    const int first = a[g.member], held = na[g.member];
    int ahead = -1;
    if (d.family == kBatchMvn) {
      const int a0 = at.y * d.ct, nc = min(d.ct, held - a0);
      const float* X = PHASE == 0 ? q : u;
      float* out = PHASE == 0 ? u : grad;
      if (d.ct == 64)
        run_mvn<PHASE, 64, 8>(d, g.ob * kOB, act, first + a0, nc, coff, X, out, part, logp,
                              smem);
      else
        run_mvn<PHASE, 32, 4>(d, g.ob * kOB, act, first + a0, nc, coff, X, out, part, logp,
                              smem);
    } else if (PHASE == 0) {
      const int a0 = at.y * d.ct;
      // These tiles are short, and last in the list: the next one is asked for first.
      if (threadIdx.x == 0) ahead = atomicAdd(next, 1);
      hier_tile(d, act, first + a0, min(d.ct, held - a0), coff, q, logp, grad);
    }
    if (threadIdx.x == 0)
      taken[turn] = (int)gridDim.x + (ahead >= 0 ? ahead : atomicAdd(next, 1));
    __syncthreads();   // every thread is done with shared memory
    tile = taken[turn];
  }
}

__global__ void iota_kernel(int* idx, int n, int* count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) idx[i] = i;
  if (i == 0) *count = n;
}

class BatchTarget final : public Target {
 public:
  BatchTarget(gbm_context* ctx, const ::gbm_batch_member* m, int64_t count) : ctx_(ctx) {
    T_ = (int)count;
    std::vector<int64_t> coff;
    std::vector<int> cdim;
    hdesc_.resize(T_);
    int64_t elems = 0, parts = 0;
    int chains = 0, dmax = 0;
    int64_t hier_chains = 0;
    for (int t = 0; t < T_; ++t)
      if (m[t].family != kBatchMvn) hier_chains += m[t].chains;
    for (int t = 0; t < T_; ++t) {
      BDesc& d = hdesc_[t];
      d = BDesc{};
      d.family = m[t].family;
      d.dim = (int)(m[t].family == kBatchMvn ? m[t].dim : m[t].dim + 2);
      d.c_begin = chains;
      d.c_end = chains + (int)m[t].chains;
      d.ct = d.family == kBatchMvn ? 64 : hier_tile_chains(hier_chains, d.dim, ctx->num_sms);
      d.p_begin = parts;
      owned_.emplace_back(new Owned());
      Owned& o = *owned_.back();
      if (d.family == kBatchMvn) {
        o.a.reserve(sizeof(float) * d.dim);
        o.b.reserve(mvn_factor_bytes(d.dim));
        GBM_CUDA(cudaMemcpyAsync(o.a.ptr, m[t].loc, sizeof(float) * d.dim,
                                 cudaMemcpyDeviceToDevice, ctx->stream));
        d.mvn = mvn_factor(m[t].scale_tril_inv, o.a.as<float>(), d.dim, m[t].log_normalizer,
                           o.b.as<float>(), ctx->stream);
        parts += (int64_t)m[t].chains * mvn_parts(d.dim);
      } else {
        const int J = d.dim - 2;
        o.a.reserve(sizeof(float) * J);
        o.b.reserve(sizeof(float) * J);
        GBM_CUDA(cudaMemcpyAsync(o.a.ptr, m[t].group_y, sizeof(float) * J,
                                 cudaMemcpyDeviceToDevice, ctx->stream));
        GBM_CUDA(cudaMemcpyAsync(o.b.ptr, m[t].group_sigma, sizeof(float) * J,
                                 cudaMemcpyDeviceToDevice, ctx->stream));
        d.y = o.a.as<float>();
        d.sigma = o.b.as<float>();
        d.mu_scale = m[t].mu_scale;
        d.tau_scale = m[t].tau_scale;
        std::vector<float> hs(J);
        GBM_CUDA(cudaMemcpyAsync(hs.data(), m[t].group_sigma, sizeof(float) * J,
                                 cudaMemcpyDeviceToHost, ctx->stream));
        GBM_CUDA(cudaStreamSynchronize(ctx->stream));
        // Normaliser of the HalfCauchy / Normal priors and the likelihood.
        const double log2pi = log(2.0 * M_PI);
        double c = log(2.0 / M_PI) - log((double)d.mu_scale) - log((double)d.tau_scale) -
                   0.5 * (1.0 + 2.0 * (double)J) * log2pi;
        for (int j = 0; j < J; ++j) c -= log((double)hs[j]);
        d.hconst = c;
      }
      for (int c = 0; c < (int)m[t].chains; ++c) {
        coff.push_back(elems);
        cdim.push_back(d.dim);
        elems += d.dim;
      }
      chains += (int)m[t].chains;
      dmax = std::max(dmax, d.dim);
    }
    C_ = chains;
    E_ = elems;
    dim = dmax;
    set_chain_models(ctx);
    coff_.reserve(sizeof(int64_t) * C_);
    cdim_.reserve(sizeof(int) * C_);
    GBM_CUDA(cudaMemcpyAsync(coff_.ptr, coff.data(), sizeof(int64_t) * C_,
                             cudaMemcpyHostToDevice, ctx->stream));
    GBM_CUDA(cudaMemcpyAsync(cdim_.ptr, cdim.data(), sizeof(int) * C_, cudaMemcpyHostToDevice,
                             ctx->stream));
    desc_.reserve(sizeof(BDesc) * T_);
    u_.reserve(sizeof(float) * (size_t)E_);
    part_.reserve(sizeof(double) * (size_t)std::max<int64_t>(parts, 1));
    make_order(0, &order_[0]);
    make_order(1, &order_[1]);
    sched_.reserve(sizeof(int) * (size_t)(2 * T_ + 4));
    all_.reserve(sizeof(int) * (size_t)(C_ + 1));
    iota_kernel<<<(C_ + 255) / 256, 256, 0, ctx->stream>>>(all_.as<int>(), C_,
                                                           all_.as<int>() + C_);
    GBM_CUDA(cudaGetLastError());
    sms_ = ctx->num_sms;
    prepare_phase<0>();
    prepare_phase<1>();
    upload();
    GBM_CUDA(cudaStreamSynchronize(ctx->stream));
    autotune();
  }

  size_t workspace_bytes(int64_t) const override { return 256; }
  const int64_t* ragged_offsets() const override { return coff_.as<int64_t>(); }
  const int* ragged_dims() const override { return cdim_.as<int>(); }
  int64_t ragged_chains() const override { return C_; }
  int64_t ragged_elements() const override { return E_; }
  int launches_per_eval(int64_t) const override { return 3; }
  const ChainModels* chain_models() const override {
    return models_.ptr ? &chain_models_ : nullptr;
  }

  // All chains (the direct log_prob_and_grad call): q, grad ragged.
  void eval(const float* q, int, const int*, int, double* logp, float* grad, int, void*,
            cudaStream_t s) override {
    int* idx = all_.as<int>();
    eval_active(q, idx, idx + C_, logp, grad, nullptr, s);
  }

  void eval_active(const float* q, const int* act, const int* act_count, double* logp,
                   float* grad, void*, cudaStream_t s) override {
    int *a = sched_.as<int>(), *na = a + T_, *totals = a + 2 * T_, *next = totals + 2;
    const BDesc* d = desc_.as<BDesc>();
    const Group *g0 = order_[0].groups.as<Group>(), *g1 = order_[1].groups.as<Group>();
    int2 *t0 = order_[0].tiles.as<int2>(), *t1 = order_[1].tiles.as<int2>();
    batch_schedule_kernel<<<dim3(2, sched_blocks_), 1024, 0, s>>>(
        d, T_, act, act_count, g0, g1, order_[0].count, order_[1].count, a, na, t0, t1, totals, next);
    batch_phase_kernel<0><<<grid_[0], kThreads, PhaseLaunch<0>::kSmem, s>>>(
        d, g0, t0, totals, next, sms_, act, a, na, coff_.as<int64_t>(), q, u_.as<float>(), grad,
        part_.as<double>(), logp);
    if (order_[1].count > 0)
      batch_phase_kernel<1>
          <<<grid_[1], kThreads * PhaseLaunch<1>::kGroups, PhaseLaunch<1>::kSmem, s>>>(
              d, g1, t1, totals + 1, next + 1, sms_, act, a, na, coff_.as<int64_t>(), q,
              u_.as<float>(), grad, part_.as<double>(), logp);
    GBM_CUDA(cudaGetLastError());
  }

  double flops(int64_t) const override {
    double f = 0.0;
    for (const BDesc& d : hdesc_) {
      const double n = d.c_end - d.c_begin;
      f += d.family == kBatchMvn ? 2.0 * d.dim * (double)d.dim * n : 10.0 * (d.dim - 2) * n;
    }
    return f;
  }
  double bytes(int64_t) const override {
    double b = 0.0;
    for (const BDesc& d : hdesc_) {
      const double n = d.c_end - d.c_begin;
      b += d.family == kBatchMvn ? 4.0 * d.dim * (double)d.dim + 8.0 * n * d.dim + 8.0 * n
                                 : 8.0 * (d.dim - 2) + 8.0 * n * d.dim + 8.0 * n;
    }
    return b;
  }

  // Chain-tile width chosen for each size class of D (0 if the class is empty).
  void schedule(int32_t* ct) const {
    for (int k = 0; k < kClasses; ++k) ct[k] = chosen_[k];
  }

 private:
  struct Owned {
    DeviceBuffer a, b;
  };

  // As many CTAs as are resident at once, whole stretches of the SMs.
  template <int PHASE>
  void prepare_phase() {
    constexpr int threads = kThreads * PhaseLaunch<PHASE>::kGroups;
    GBM_CUDA(cudaFuncSetAttribute(batch_phase_kernel<PHASE>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  PhaseLaunch<PHASE>::kSmem));
    int per_sm = 0;
    GBM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_phase_kernel<PHASE>,
                                                           threads, PhaseLaunch<PHASE>::kSmem));
    grid_[PHASE] = std::max(1, per_sm) * sms_;
  }

  struct Order {
    int count = 0;              // groups
    DeviceBuffer groups, tiles;
  };

  // The groups of a phase, those with the longest sums first (hierarchical
  // tiles, short, at the end of phase 0), and room for their tiles.
  void make_order(int phase, Order* order) {
    std::vector<Group> groups;
    size_t tiles = 0;
    for (int t = 0; t < T_; ++t) {
      const BDesc& d = hdesc_[t];
      const int chains = d.c_end - d.c_begin;
      if (d.family == kBatchMvn) {
        const int nob = (d.dim + kOB - 1) / kOB;
        for (int ob = 0; ob < nob; ++ob) groups.push_back(Group{t, ob});
        tiles += (size_t)nob * ((chains + 31) / 32);
      } else if (phase == 0) {
        groups.push_back(Group{t, 0});
        tiles += (size_t)(chains + d.ct - 1) / d.ct;
      }
    }
    auto length = [&](const Group& g) {
      const BDesc& d = hdesc_[g.member];
      if (d.family != kBatchMvn) return 0;
      return phase == 0 ? std::min(d.dim, (g.ob + 1) * kOB) : d.dim - g.ob * kOB;
    };
    std::stable_sort(groups.begin(), groups.end(),
                     [&](const Group& x, const Group& y) { return length(x) > length(y); });
    order->count = (int)groups.size();
    const int blocks = (int)std::min<size_t>((tiles + 8191) / 8192, (size_t)ctx_->num_sms / 2);
    sched_blocks_ = std::max(sched_blocks_, blocks);
    order->groups.reserve(sizeof(Group) * std::max<size_t>(groups.size(), 1));
    order->tiles.reserve(sizeof(int2) * std::max<size_t>(tiles, 1));
    GBM_CUDA(cudaMemcpyAsync(order->groups.ptr, groups.data(), sizeof(Group) * groups.size(),
                             cudaMemcpyHostToDevice, ctx_->stream));
    GBM_CUDA(cudaStreamSynchronize(ctx_->stream));   // the vector is this call's
  }

  // The hierarchical members whose chains a warp holds (kChainMaxDim elements).
  void set_chain_models(gbm_context* ctx) {
    const std::vector<double> table = chain_log_table();
    table_.reserve(sizeof(double) * table.size());
    std::vector<HierModel> models(T_);
    std::vector<int> model_of(C_, -1);
    int max_dim = 0, held = 0;
    for (int t = 0; t < T_; ++t) {
      const BDesc& d = hdesc_[t];
      if (d.family != kBatchHier || d.dim > kChainMaxDim) continue;
      models[t] = HierModel{d.y, d.sigma, d.mu_scale, d.tau_scale, d.hconst, table_.as<double>()};
      std::fill(model_of.begin() + d.c_begin, model_of.begin() + d.c_end, t);
      max_dim = std::max(max_dim, d.dim);
      held += d.c_end - d.c_begin;
    }
    if (held == 0) return;
    GBM_CUDA(cudaMemcpyAsync(table_.ptr, table.data(), sizeof(double) * table.size(),
                             cudaMemcpyHostToDevice, ctx->stream));
    models_.reserve(sizeof(HierModel) * T_);
    model_of_.reserve(sizeof(int) * C_);
    GBM_CUDA(cudaMemcpyAsync(models_.ptr, models.data(), sizeof(HierModel) * T_,
                             cudaMemcpyHostToDevice, ctx->stream));
    GBM_CUDA(cudaMemcpyAsync(model_of_.ptr, model_of.data(), sizeof(int) * C_,
                             cudaMemcpyHostToDevice, ctx->stream));
    GBM_CUDA(cudaStreamSynchronize(ctx->stream));   // the vectors are this call's
    chain_models_ = ChainModels{models_.as<HierModel>(), model_of_.as<int>(), max_dim,
                                held == C_};
  }

  void upload() {
    GBM_CUDA(cudaMemcpyAsync(desc_.ptr, hdesc_.data(), sizeof(BDesc) * T_,
                             cudaMemcpyHostToDevice, ctx_->stream));
  }

  // For each size class of D: time a full evaluation of every chain with
  // that class's MVN tiles at 32 and at 64 chains and keep the faster.
  void autotune() {
    cudaStream_t s = ctx_->stream;
    double* lp = nullptr;
    float* g = nullptr;
    DeviceBuffer qb, lb, gb;
    qb.reserve(sizeof(float) * (size_t)E_);
    lb.reserve(sizeof(double) * (size_t)C_);
    gb.reserve(sizeof(float) * (size_t)E_);
    GBM_CUDA(cudaMemsetAsync(qb.ptr, 0, sizeof(float) * (size_t)E_, s));
    lp = lb.as<double>();
    g = gb.as<float>();
    cudaEvent_t e0, e1;
    GBM_CUDA(cudaEventCreate(&e0));
    GBM_CUDA(cudaEventCreate(&e1));
    for (int k = 0; k < kClasses; ++k) {
      chosen_[k] = 0;
      bool any = false;
      for (const BDesc& d : hdesc_) any |= d.family == kBatchMvn && size_class(d.dim) == k;
      if (!any) continue;
      float best = 1e30f;
      for (int ct : {32, 64}) {
        for (BDesc& d : hdesc_)
          if (d.family == kBatchMvn && size_class(d.dim) == k) d.ct = ct;
        upload();
        eval(qb.as<float>(), 0, nullptr, 0, lp, g, 0, nullptr, s);   // warm-up
        GBM_CUDA(cudaEventRecord(e0, s));
        for (int r = 0; r < 3; ++r) eval(qb.as<float>(), 0, nullptr, 0, lp, g, 0, nullptr, s);
        GBM_CUDA(cudaEventRecord(e1, s));
        GBM_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        GBM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best) {
          best = ms;
          chosen_[k] = ct;
        }
      }
      for (BDesc& d : hdesc_)
        if (d.family == kBatchMvn && size_class(d.dim) == k) d.ct = chosen_[k];
    }
    upload();
    GBM_CUDA(cudaStreamSynchronize(s));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }

  gbm_context* ctx_;
  int T_ = 0, C_ = 0, sms_ = 0, grid_[2] = {0, 0}, sched_blocks_ = 1;
  int64_t E_ = 0;
  int chosen_[kClasses] = {0, 0, 0, 0};
  std::vector<BDesc> hdesc_;
  Order order_[2];
  std::vector<std::unique_ptr<Owned>> owned_;
  DeviceBuffer desc_, coff_, cdim_, u_, part_, sched_, all_, models_, model_of_, table_;
  ChainModels chain_models_{};
};

}  // namespace

std::unique_ptr<Target> make_batch(gbm_context* ctx, const ::gbm_batch_member* m,
                                   int64_t count) {
  return std::unique_ptr<Target>(new BatchTarget(ctx, m, count));
}

bool batch_schedule(const Target* t, int32_t* ct) {
  const auto* b = dynamic_cast<const BatchTarget*>(t);
  if (!b) return false;
  b->schedule(ct);
  return true;
}

}  // namespace gbm
