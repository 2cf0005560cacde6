// Whole leapfrog trajectories of a small FP32 logistic regression in one launch.
//
// A cluster of CTAs holds all of X in shared memory, feature-major, and carries a
// few chains through every step of their trajectories: no launch, no partial in
// global memory and no other cluster is waited for between two gradients.  A step:
//   residuals  a thread takes four consecutive rows of a chain: z, then R (to
//              shared memory) and, at the last step, the likelihood terms;
//   products   a thread takes a row split and a feature: sum_r R[r] x[r], the
//              chains of the cluster side by side;
//   update     a thread takes a chain and a feature: the splits' sums (the other
//              CTAs' over distributed shared memory), the prior, kick and drift,
//              in every CTA of the cluster alike.
// Splits, orders of addition and roundings are those of logreg_f32_kernel and the
// split reduction, so a trajectory is theirs to the bit.
//
// What bounds it: latency (a split's 64 dependent FMAs a feature, the z of four
// rows, three barriers).  A step of 1000 x 25, 64 chains takes 3.0 us (three launches
// a step: 30), of 64 x 2, 16 chains 1.5 (20), of 2000 x 60, 128 chains on clusters
// of four 8.9 (40), of 2000 x 100, 64 chains 21 (49).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "logreg_f32_math.cuh"
#include "split_reduce.cuh"
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr int kLeapThreads = 512;
constexpr int kLeapTile = 64;              // rows of logreg_f32_kernel's tiles
constexpr int kLeapMaxCluster = 8;
// Clusters are launched up to four times as many as run at once: 4000 x 10, 1024
// chains 25 us a step, three launches a step 34.  From there on those, which fill
// the GPU, catch up.
constexpr int kLeapWaves = 4;
constexpr int64_t kLeapSmem = 227 * 1024;

// What a launch holds in shared memory, in floats (64 bits: leap_shape asks for any
// number of rows).
struct LeapShape {
  int K, G;            // CTAs of a cluster, chains of a cluster
  int S, row_tiles;    // row splits of the whole, row tiles of the whole
  int rowpad;          // row stride of X and R, 4 modulo 32 (16-byte loads of
                       // neighbouring features without conflicts)
  int smax;            // most splits of a CTA
  int D;
  __host__ __device__ int64_t x() const { return 0; }
  __host__ __device__ int64_t y() const { return (int64_t)D * rowpad; }
  __host__ __device__ int64_t r() const { return y() + rowpad; }
  __host__ __device__ int64_t like() const { return r() + (int64_t)G * rowpad; }
  __host__ __device__ int64_t part() const { return like() + (int64_t)G * (rowpad / 4); }
  __host__ __device__ int64_t q() const { return part() + (int64_t)2 * smax * G * D; }
  __host__ __device__ int64_t p() const { return q() + (int64_t)G * D; }
  __host__ __device__ int64_t sums() const { return (p() + (int64_t)G * D + 1) / 2 * 2; }
  __host__ __device__ int64_t bytes() const {
    return 4 * (sums() + 2 * G * (1 + kLeapThreads / 32));
  }
};

// First row tile of split s.
__host__ __device__ inline int leap_tile(const LeapShape& h, int s) {
  return (int)((long long)s * h.row_tiles / h.S);
}
__host__ __device__ inline int leap_split(const LeapShape& h, int rank) {
  return rank * h.S / h.K;
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ double ld_cluster_f64(uint32_t addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

// X2, ym: logreg_f32.cu's layout.  q, p, g: [C][ld]; logp [C].
template <int G>
__global__ void __launch_bounds__(kLeapThreads, 1)
logreg_leapfrog_kernel(LeapShape h, const float* __restrict__ X2, const float* __restrict__ ym,
                       int N, int Dp, int C, int steps, const float* __restrict__ eps,
                       int per_chain, float inv_var, double log_norm,
                       const double* __restrict__ lin, float* __restrict__ q,
                       float* __restrict__ p, float* __restrict__ g, double* __restrict__ logp,
                       int ld) {
  extern __shared__ __align__(16) float leap_smem[];
  float* smem = leap_smem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = h.D;
  const int rank = h.K > 1 ? (int)tc::cluster_ctarank() : 0;
  const int c0 = (int)blockIdx.x / h.K * G, held = min(G, C - c0);
  const int s0 = leap_split(h, rank), s1 = leap_split(h, rank + 1);
  const int t0 = leap_tile(h, s0), rows = (leap_tile(h, s1) - t0) * kLeapTile, quads = rows / 4;
  float *Xs = smem + h.x(), *Ys = smem + h.y(), *Rs = smem + h.r(), *Ls = smem + h.like();
  float *Ps = smem + h.part(), *Qs = smem + h.q(), *Ms = smem + h.p();
  double* sums = reinterpret_cast<double*>(smem + h.sums());   // [G], then [warps][G]
  auto sync = [&]() {
    if (h.K > 1)
      tc::cluster_sync();
    else
      __syncthreads();
  };

  // X of this CTA's rows, feature-major; chains past the last are zero.
  {
    const float2* src = reinterpret_cast<const float2*>(X2) + (size_t)t0 * (kLeapTile / 2) * Dp;
    for (int i = tid; i < rows / 2 * D; i += kLeapThreads) {
      const int pair = i / D, d = i - pair * D;
      const float2 v = src[(size_t)pair * Dp + d];
      *reinterpret_cast<float2*>(Xs + d * h.rowpad + 2 * pair) = v;
    }
    for (int i = tid; i < rows; i += kLeapThreads) Ys[i] = ym[(size_t)t0 * kLeapTile + i];
    for (int i = tid; i < G * D; i += kLeapThreads) {
      const int c = i / D, d = i - c * D;
      const size_t at = (size_t)(c0 + c) * ld + d;
      Qs[i] = c < held ? q[at] : 0.f;
      Ms[i] = c < held ? p[at] : 0.f;
    }
  }
  __syncthreads();

  for (int step = 0; step < steps; ++step) {
    const bool last = step + 1 == steps;
    // ---- residuals ----
    for (int i = tid; i < quads * G; i += kLeapThreads) {
      const int c = i / quads, quad = i - c * quads;
      const float* xp = Xs + 4 * quad;
      const float* qp = Qs + c * D;
      float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int d = 0; d < D; ++d) {
        const float4 x = *reinterpret_cast<const float4*>(xp + d * h.rowpad);
        const float b = qp[d];
        z[0] = fmaf(x.x, b, z[0]);
        z[1] = fmaf(x.y, b, z[1]);
        z[2] = fmaf(x.z, b, z[2]);
        z[3] = fmaf(x.w, b, z[3]);
      }
      const float4 y4 = *reinterpret_cast<const float4*>(Ys + 4 * quad);
      const float yr[4] = {y4.x, y4.y, y4.z, y4.w};
      const int nvalid = N - t0 * kLeapTile - 4 * quad;
      float r[4], sabs = 0.f, prod = 1.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) f32_residual(z[k], yr[k], k < nvalid, sabs, prod, r[k]);
      *reinterpret_cast<float4*>(Rs + c * h.rowpad + 4 * quad) = make_float4(r[0], r[1], r[2], r[3]);
      if (last) Ls[c * (h.rowpad / 4) + quad] = f32_like(sabs, prod);
    }
    __syncthreads();
    // ---- products ----
    float* part = Ps + (step & 1) * h.smax * G * D;
    for (int i = tid; i < (s1 - s0) * D; i += kLeapThreads) {
      const int s = i / D, f = i - s * D;
      const int a = (leap_tile(h, s0 + s) - t0) * kLeapTile;
      const int b = (leap_tile(h, s0 + s + 1) - t0) * kLeapTile;
      const float* xp = Xs + f * h.rowpad;
      float acc[G];
#pragma unroll
      for (int c = 0; c < G; ++c) acc[c] = 0.f;
#pragma unroll 4
      for (int r = a; r < b; r += 4) {
        const float4 x = *reinterpret_cast<const float4*>(xp + r);
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(Rs + c * h.rowpad + r);
          acc[c] = fmaf(v.x, x.x, acc[c]);
          acc[c] = fmaf(v.y, x.y, acc[c]);
          acc[c] = fmaf(v.z, x.z, acc[c]);
          acc[c] = fmaf(v.w, x.w, acc[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < G; ++c) part[(s * G + c) * D + f] = acc[c];
    }
    sync();
    // ---- update ----
    for (int i = tid; i < held * D; i += kLeapThreads) {
      const int c = i / D, f = i - c * D;
      // Splits [a, b) in order, from the CTAs that hold them.
      auto add = [&](int a, int b) {
        float acc = 0.f;
        int k = 0;
        for (int s = a; s < b;) {
          while (leap_split(h, k + 1) <= s) ++k;
          const int first = leap_split(h, k), end = min(b, leap_split(h, k + 1));
          const float* mine = part + ((s - first) * G + c) * D + f;
          if (h.K == 1) {
#pragma unroll 8
            for (; s < end; ++s, mine += G * D) acc += *mine;
          } else {
            uint32_t at = tc::map_to_rank(tc::smem_u32(mine), (uint32_t)k);
            for (; s < end; s += 8, at += 32 * G * D) {
              float v[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) v[u] = s + u < end ? ld_cluster_f32(at + 4 * u * G * D) : 0.f;
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (s + u < end) acc += v[u];
            }
            s = end;
          }
        }
        return acc;
      };
      float acc;
      if (h.S <= kOrdered) {
        acc = add(0, h.S);
      } else {
        acc = add(0, h.S / kReduceGroups);
        for (int j = 1; j < kReduceGroups; ++j)
          acc += add(j * h.S / kReduceGroups, (j + 1) * h.S / kReduceGroups);
      }
      const float qv = Qs[i], grad = acc - qv * inv_var;
      const size_t at = (size_t)(c0 + c) * ld + f;
      if (last) {
        if (rank == 0) {
          g[at] = grad;
          q[at] = qv;
          p[at] = Ms[i];
        }
      } else {
        const float e = eps[per_chain ? c0 + c : 0];
        const float ph = Ms[i] + e * grad;
        Ms[i] = ph;
        Qs[i] = qv + e * ph;
      }
    }
    __syncthreads();
  }

  // ---- log-density at the last state ----
  // Each (split, row of quads) adds its tiles in FP32 with Kahan's correction, the
  // rest in float64.
  double like[G];
#pragma unroll
  for (int c = 0; c < G; ++c) like[c] = 0.0;
  for (int i = tid; i < (s1 - s0) * 16; i += kLeapThreads) {
    const int s = i >> 4, ty = i & 15;
    const int a = leap_tile(h, s0 + s) - t0, b = leap_tile(h, s0 + s + 1) - t0;
#pragma unroll
    for (int c = 0; c < G; ++c) {
      float lsum = 0.f, lcomp = 0.f;
      for (int t = a; t < b; ++t) kahan_add(Ls[c * (h.rowpad / 4) + 16 * t + ty], lsum, lcomp);
      like[c] += (double)lsum - (double)lcomp;
    }
  }
#pragma unroll
  for (int c = 0; c < G; ++c) {
    const double s = warp_sum(like[c]);
    if (lane == 0) sums[G + warp * G + c] = s;
  }
  __syncthreads();
  if (tid < G) {
    double s = 0.0;
    for (int w = 0; w < kLeapThreads / 32; ++w) s += sums[G + w * G + tid];
    sums[tid] = s;
  }
  sync();
  if (rank == 0 && warp < held) {
    const int c = warp;
    double t = 0.0;
    for (int d = lane; d < D; d += 32) {
      const double qd = (double)Qs[c * D + d];
      t += lin[d] * qd - 0.5 * (double)inv_var * qd * qd;
    }
    t = warp_sum(t);
    if (lane == 0) {
      for (int k = 0; k < h.K; ++k)
        t += h.K > 1 ? ld_cluster_f64(tc::map_to_rank(tc::smem_u32(sums + c), (uint32_t)k))
                     : sums[c];
      logp[c0 + c] = t + (double)D * log_norm;
    }
  }
  if (h.K > 1) tc::cluster_sync();   // rank 0 has read the others' sums
}

// The launch for C chains, if X fits a cluster's shared memory and the clusters
// the GPU: false otherwise.  The fewest waves first, then the smallest cluster (no
// exchange at all with one CTA), then the fewest chains a cluster.
inline bool leap_shape(int64_t N, int D, int C, int grid_max, int chain_tile, LeapShape* out) {
  LeapShape h;
  h.D = D;
  h.row_tiles = (int)((N + kLeapTile - 1) / kLeapTile);
  const int g = work_grid(grid_max, C, chain_tile, N, kMinSplitRows);
  h.S = split_count(C, chain_tile, kLeapTile, g, (int)N);
  for (int waves = 1; waves <= kLeapWaves; waves *= 2)
    for (h.K = 1; h.K <= kLeapMaxCluster; h.K *= 2) {
      int tiles = 0;
      h.smax = 0;
      for (int k = 0; k < h.K; ++k) {
        const int a = leap_split(h, k), b = leap_split(h, k + 1);
        h.smax = std::max(h.smax, b - a);
        tiles = std::max(tiles, leap_tile(h, b) - leap_tile(h, a));
      }
      h.rowpad = (tiles * kLeapTile + 31) / 32 * 32 + 4;
      for (h.G = 1; h.G <= 4; h.G *= 2)
        if ((int64_t)((C + h.G - 1) / h.G) * h.K <= (int64_t)waves * grid_max &&
            h.bytes() <= kLeapSmem) {
          *out = h;
          return true;
        }
    }
  return false;
}

// Once before the launches.
template <int G>
void prepare_leapfrogs() {
  GBM_CUDA(cudaFuncSetAttribute(logreg_leapfrog_kernel<G>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLeapSmem));
}

template <int G>
void launch_leapfrogs(const LeapShape& h, const float* X2, const float* ym, int N, int Dp, int C,
                      int steps, const float* eps, int per_chain, float inv_var, double log_norm,
                      const double* lin, float* q, float* p, float* g, double* logp, int ld,
                      cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((C + G - 1) / G * h.K));
  cfg.blockDim = dim3(kLeapThreads);
  cfg.dynamicSmemBytes = (size_t)h.bytes();
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)h.K;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  GBM_CUDA(cudaLaunchKernelEx(&cfg, logreg_leapfrog_kernel<G>, h, X2, ym, N, Dp, C, steps, eps,
                              per_chain, inv_var, log_norm, lin, q, p, g, logp, ld));
}

}  // namespace
}  // namespace gbm
