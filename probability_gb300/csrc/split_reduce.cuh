// Deterministic sum of per-split partial results of a row-split logistic
// regression evaluation, plus the Normal(0, s) prior.
//
// Layout written by the partial kernels: lpart[S][n] (float64) and
// gpart[S][n][D] (float32), where S = number of row splits for n chains:
//   S = clamp(grid / ceil(n / ct), 1, ceil(N / nt)).
// One block per chain and 128 features (or several chains of up to 64 features, where
// there are many): a thread owns a feature and adds up to
// kOrdered splits in index order, 16 loads in flight; with more splits, groups of
// 128 threads add a range of them each and the ranges are added in order.  The
// log-density terms (likelihood partials, prior, linear part) are combined per
// lane by the last warp of a chain's first block and summed by one float64 warp
// reduction.  The order depends only on S, D and the launch, so results are
// reproducible.
//
// What bounds it: the latency of the partials' loads (L2), so the loads of a
// chain are spread over threads instead of over rounds of one warp.  Measured
// with the partial kernel: 12,007 x 173 BF16, 77 chains (94 splits) 37.2 us with
// a warp per chain, 28.7 with a block, 26.3 so; 12,289 x 601 FP32, 99 chains (50
// splits) 95.2 with a block for all features, 90.6 so; a step of three launches at
// 1000 x 25, 64 chains 40.8 with a warp, 38.2 with a block; 1024 chains (19 splits)
// the same (four groups there: 10 us more).
// `lin` (optional, float64 [D]) adds lin . q_c to each chain's log-density:
// the tensor-core kernels leave the linear part sum_r (y_r - 1/2) z_rc of the
// Bernoulli log-likelihood to this pass as (X^T (y - 1/2)) . q_c, exact in
// float64.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace gbm {

constexpr int kOrdered = 32;               // splits one thread adds
constexpr int kReduceGroups = 4;           // groups of 128 threads when there may be more
// Chains from which a block takes several of up to 64 features: those of fewer are
// all in flight at once whatever the block, and more wait for issue and the FP64
// pipe, which idle warps take their share of (50 x 4, 19,456 chains: 39.5 us an
// evaluation with a block a chain, 31 so; 1000 x 25, 4096: 37.5 and 35.4).
constexpr int kPackedChains = 2048;

// Chains of one launch.  A launch covers at most grid * ct chains (one work
// item per CTA); larger batches are evaluated as consecutive chunks of
// `c_lim` chains starting at chain `c_base` (pointers offset by the caller).
// Chunk k sees min(max(n - c_base, 0), c_lim) chains of the n in *n_dev.
__host__ __device__ __forceinline__ int chunk_count(int n, int c_base, int c_lim) {
  const int m = n - c_base;
  return m < 0 ? 0 : (m > c_lim ? c_lim : m);
}

// CTAs (or CTA pairs) of one launch: at most grid_max, and no more than the
// call's chain tiles times the row splits that keep at least min_rows rows
// each, so no CTA is launched only to find no work.  With min_rows = 64 (the
// smallest row tile) the split counts are those of the full grid: a small,
// latency-bound evaluation keeps one row tile per CTA.  Kernels and the split
// reduction derive the split count from the grid they are given, so passing
// this value to both keeps them consistent.
inline int work_grid(int grid_max, int64_t chains, int ct, int64_t N, int64_t min_rows) {
  const int64_t tiles = (chains + ct - 1) / ct;
  const int64_t s_cap = N / min_rows > 1 ? N / min_rows : 1;
  int64_t g = tiles * s_cap;
  if (g > grid_max) g = grid_max;
  return g < 1 ? 1 : (int)g;
}

constexpr int64_t kMinSplitRows = 64;

namespace {

__host__ __device__ __forceinline__ int split_count(int n, int ct, int nt, int grid, int N) {
  const int tiles = (n + ct - 1) / ct;
  if (tiles == 0) return 0;
  int s = grid / tiles;
  s = s < 1 ? 1 : s;
  const int row_tiles = (N + nt - 1) / nt;
  return s > row_tiles ? row_tiles : s;
}

// Sum of p[s * stride], s in [s0, s1), in order, U loads in flight.
template <int U>
__device__ __forceinline__ float sum_splits(const float* __restrict__ p, size_t stride, int s0,
                                            int s1) {
  float acc = 0.f;
  int s = s0;
  for (; s + U <= s1; s += U) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = p[(size_t)(s + u) * stride];
#pragma unroll
    for (int u = 0; u < U; ++u) acc += v[u];
  }
  if (s < s1) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = s + u < s1 ? p[(size_t)(s + u) * stride] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s + u < s1) acc += v[u];
  }
  return acc;
}

// F threads a chain: 128, of which there may be several groups, or 32 or 64 of a block
// of 128.
template <int F>
__global__ void __launch_bounds__(F == 128 ? 128 * kReduceGroups : 128)
split_reduce_kernel(const double* __restrict__ lpart, const float* __restrict__ gpart,
                    const float* __restrict__ Q, int ldq, const int* __restrict__ n_dev,
                    int c_base, int c_lim, int ct, int nt, int grid, int N, int D,
                    float inv_var, double half_inv_var, double dims, double log_norm,
                    const double* __restrict__ lin, int lparts,
                    double* __restrict__ logp, float* __restrict__ grad, int ldg) {
  __shared__ float range[F == 128 ? kReduceGroups - 1 : 1][F];
  const int n = n_dev ? chunk_count(*n_dev, c_base, c_lim) : c_lim;
  const int c = F == 128 ? (int)blockIdx.x : (int)(blockIdx.x * (128 / F) + threadIdx.x / F);
  if (c >= n) return;
  const int threads = F == 128 ? (int)blockDim.x : F;               // of this chain
  const int thread = F == 128 ? (int)threadIdx.x : (int)threadIdx.x % F;
  const int S = split_count(n, ct, nt, grid, N);
  const float* q = Q + (size_t)c * ldq;
  const int groups = S <= kOrdered ? 1 : max(1, threads >> 7);
  const int group = thread >> 7, first = thread & 127;
  const int d = blockIdx.y * 128 + first;
  float acc = 0.f;
  if (d < D && group < groups)
    acc = sum_splits<F == 128 ? 16 : 4>(gpart + (size_t)c * D + d, (size_t)n * D,
                     groups > 1 ? group * S / groups : 0,
                     groups > 1 ? (group + 1) * S / groups : S);
  // Per-lane log-density terms, by the last warp beside the others' sums:
  // likelihood partials lane, lane + 32, ..., then lin . q - q.q / (2 s^2) over
  // features lane, lane + 32, ...
  if (blockIdx.y == 0 && thread + 32 >= threads) {
    const int lane = threadIdx.x & 31, rows = lparts > 0 ? lparts : S;
    double t = 0.0, pr = 0.0, li = 0.0;
    constexpr int U = F == 128 ? 8 : 1, V = F == 128 ? 4 : 1;   // steps whose loads are in flight
#pragma unroll 1
    for (int j = lane; j < rows; j += 32 * U) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = u == 0 || j + 32 * u < rows ? lpart[(size_t)(j + 32 * u) * n + c] : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u == 0 || j + 32 * u < rows) t += v[u];
    }
#pragma unroll 1
    for (int f = lane; f < D; f += 32 * V) {
      float qv[V];
      double lv[V];
#pragma unroll
      for (int u = 0; u < V; ++u) {
        const bool held = u == 0 || f + 32 * u < D;
        qv[u] = held ? q[f + 32 * u] : 0.f;
        lv[u] = held && lin ? lin[f + 32 * u] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < V; ++u)
        if (u == 0 || f + 32 * u < D) {
          const double qd = (double)qv[u];
          pr += qd * qd;
          if (lin) li += lv[u] * qd;
        }
    }
    t = warp_sum(t + li - half_inv_var * pr);
    if (lane == 0) logp[c] = t + dims * log_norm;
  }
  if (groups > 1) {
    if (group > 0) range[group - 1][first] = acc;
    __syncthreads();
    if (group == 0)
      for (int g = 0; g + 1 < groups; ++g) acc += range[g][first];
  }
  if (group == 0 && d < D) grad[(size_t)c * ldg + d] = acc - q[d] * inv_var;
}

// Q, logp and grad point at chain c_base of the batch; `cap` bounds this
// chunk's chains (<= c_lim).  lparts: rows of lpart where they are not the
// splits of the gradient; n_dev NULL: c_lim chains.
void launch_split_reduce(const double* lpart, const float* gpart, const float* Q, int ldq,
                         const int* n_dev, int c_base, int c_lim, int cap, int ct, int nt,
                         int grid, int N, int D, float inv_var, double log_norm,
                         const double* lin, double* logp, float* grad, int ldg, cudaStream_t s,
                         int lparts = 0) {
  // Few chains make many splits: several threads per feature.  (A sampler's
  // active chains are fewer than cap; one thread then adds more than kOrdered.)
  const int threads = split_count(cap, ct, nt, grid, N) <= kOrdered ? 128 : 128 * kReduceGroups;
  auto go = [&](auto kernel, int per_block) {
    const dim3 blocks((unsigned)((cap + per_block - 1) / per_block), (unsigned)((D + 127) / 128));
    kernel<<<blocks, threads, 0, s>>>(lpart, gpart, Q, ldq, n_dev, c_base, c_lim, ct, nt, grid, N,
                                      D, inv_var, 0.5 * (double)inv_var, (double)D, log_norm, lin,
                                      lparts, logp, grad, ldg);
  };
  if (threads == 128 && D <= 32 && cap >= kPackedChains)
    go(split_reduce_kernel<32>, 4);
  else if (threads == 128 && D <= 64 && cap >= kPackedChains)
    go(split_reduce_kernel<64>, 2);
  else
    go(split_reduce_kernel<128>, 1);
  GBM_CUDA(cudaGetLastError());
}

}  // namespace

}  // namespace gbm
