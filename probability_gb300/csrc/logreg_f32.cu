// Fused logistic-regression log-density + gradient, FP32 CUDA cores, for up
// to 128 features (the plain FP32 form of the 1e5 x 100 workload).
//
// Mathematics (the inference_gym logistic-regression target,
// spinoffs/inference_gym/inference_gym/targets/logistic_regression.py:92-103,
// with the Bernoulli log-prob of distributions/bernoulli.py:126-140): for
// states q_c and z_rc = x_r . q_c,
//   log p(y_r | z) = y z - softplus(z) = (y - 1/2) z - |z|/2 - ln(1 + e^-|z|)
//   R_rc = y_r - sigmoid(z_rc) = (y_r - 1/2) - sign(z) (1/(1 + e^-|z|) - 1/2)
//   grad_c = X^T R_c - q_c / s^2.
// The linear part sum_r (y_r - 1/2) z_rc = (X^T (y - 1/2)) . q_c is added
// exactly (float64) by the split reduction; this kernel accumulates
// -(sum |z|/2 + sum ln(1 + e^-|z|)) and X^T R.
//
// Work decomposition: one CTA (256 threads, one per SM) owns a tile of 128
// chains and a contiguous range of 64-row tiles of X (a row split).  Per row
// tile, in FP32 on the CUDA cores:
//   phase 1  Z[64 rows][128 chains] = X_tile B^T: each thread 4 rows x 8
//            chains, K = features, 6 shared loads per 64 FMAs;
//   epilogue the log-likelihood sums and R (to shared memory);
//   phase 2  G[128 chains][Dp] += R^T X_tile: each thread 8 chains x KD
//            features (features f + 16 j), held in registers across the
//            CTA's rows, 4 + KD shared loads per 16 KD FMAs.
// X is stored on the device in row pairs, X2[N/2][Dp][2] (element (r, d) at
// ((r/2) Dp + d) 2 + r%2), zero-padded to Dp = 16 KD features and whole
// 64-row tiles, so that one 16-byte load gives phase 1 two rows x two
// features and one 8-byte load gives phase 2 two rows of one feature, and a
// row tile is one contiguous block moved by one bulk copy (cp.async.bulk)
// into a double-buffered shared-memory stage.  X is read from HBM once per
// chain tile (L2 serves the other chain tiles of the same rows).
//
// From kPairRows rows on, phase 2 runs on the tensor cores instead
// (logreg_f32_tc_kernel), beside phase 1 of the next tile: the residuals go to
// shared memory as FP16 hi + lo (of R 2^15) and X is kept as FP16 hi + lo
// (of each feature scaled to the top of FP16's range) beside its FP32 form,
//   G^T = R_lo^T X_hi + R_hi^T X_lo + R_hi^T X_hi  (M = 128 chains, K = 64 rows).
// hi + lo carries a float to 2^-23 of itself at worst (f16_rows.cuh says for which
// columns); what is left out (lo.lo) is as small.  The tensor cores truncate every
// addition to their FP32 accumulator, so a turn of at most two tiles starts from zero, the small terms of a tile
// first, and is then added in FP32 to the sum of the turns before: gradient
// error against 64 bits 1.4e-7 at 1e5 x 100 x 1024 chains (phase 2 on the CUDA
// cores: 2.9e-7).  Z, and with it the log-density, is phase 1's, bit for bit.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>

#include "engine.h"
#include "f16_rows.cuh"
#include "logreg_f32_math.cuh"
#include "logreg_leapfrog.cuh"
#include "split_reduce.cuh"
#include "tc_common.cuh"
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr int kF32CT = 128;                 // chains per tile
constexpr int kF32RT = 64;                  // rows per tile
constexpr int kF32Threads = 256;
constexpr uint64_t kF32WaitNs = 2000000000ull;   // 2 s bound on every wait
constexpr int kF32TimeoutCode = 4;                // error word: bulk copy never landed

template <int KD>
struct F32Layout {
  static constexpr int kDp = 16 * KD;
  static constexpr int kBt = 0;                               // [Dp][128] float
  static constexpr int kXStage = kF32RT * kDp * 4;            // one row tile of X2
  static constexpr int kX = kBt + kDp * kF32CT * 4;           // 2 stages
  static constexpr int kY = kX + 2 * kXStage;                 // 2 x [64] float (y - 1/2)
  static constexpr int kR = kY + 2 * kF32RT * 4;              // [64][128] float
  static constexpr int kBar = kR + kF32RT * kF32CT * 4;       // 2 mbarriers + flag
  static constexpr int kBytes = kBar + 64;
  static_assert(16 * kF32CT * 8 <= kF32RT * kF32CT * 4, "reduction scratch fits R");
  static_assert(kBytes <= 232448, "shared memory over the sm_103a limit");
};

__host__ __device__ inline int f32_splits(int n, int grid, int row_tiles) {
  const int tiles = (n + kF32CT - 1) / kF32CT;
  if (tiles == 0) return 0;
  int s = grid / tiles;
  s = s < 1 ? 1 : s;
  return s > row_tiles ? row_tiles : s;
}

__device__ __forceinline__ float4 lds4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}

// Phase 1 of one thread: z[i][c] = x_i . B_c over dk features (even) for its
// four rows (row pairs xa and xa + pair) and eight chains (bp and bp + 64), K
// in order.
__device__ __forceinline__ void f32_phase1(float (&z)[4][8], const float* xa, int pair,
                                           const float* bp, int dk) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 8; ++c) z[i][c] = 0.f;
  const float* xb = xa + pair;
  // Register double buffering: the next feature pair's six loads are in
  // flight while this pair's 64 FMAs issue (the last iteration re-reads
  // its own pair instead of reading past the tile).
  float4 u = lds4(xa), v = lds4(xb);   // x(r0,d) x(r1,d) x(r0,d+1) x(r1,d+1); rows r2, r3
  float4 b0 = lds4(bp), b1 = lds4(bp + 64), b2 = lds4(bp + kF32CT), b3 = lds4(bp + kF32CT + 64);
#pragma unroll 2
  for (int d = 0; d < dk; d += 2) {
    const int dn = d + 2 < dk ? d + 2 : d;
    const float4 un = lds4(xa + 2 * dn), vn = lds4(xb + 2 * dn);
    const float4 b0n = lds4(bp + dn * kF32CT), b1n = lds4(bp + dn * kF32CT + 64);
    const float4 b2n = lds4(bp + (dn + 1) * kF32CT), b3n = lds4(bp + (dn + 1) * kF32CT + 64);
    const float xr0[4] = {u.x, u.y, v.x, v.y};
    const float xr1[4] = {u.z, u.w, v.z, v.w};
    const float bb0[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    const float bb1[8] = {b2.x, b2.y, b2.z, b2.w, b3.x, b3.y, b3.z, b3.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c) z[i][c] = fmaf(xr1[i], bb1[c], fmaf(xr0[i], bb0[c], z[i][c]));
    u = un; v = vn; b0 = b0n; b1 = b1n; b2 = b2n; b3 = b3n;
  }
}

// Phase 1 of one thread over NT row tiles (`tile` floats apart): its four rows
// of each and eight chains, two chains to an instruction (fma.rn.f32x2: the
// same roundings); z[4 t + i] are row i of tile t.  With two tiles a fragment of
// B^T feeds 16 rows' worth of loads' FMAs: 107 FMAs a clock and SM where the
// 4 x 8 tile above gets 79 (of 128; measured in a loop of nothing else).
template <int NT>
__device__ __forceinline__ void f32_phase1_pairs(float2 (&z)[8][4], const float* xp, int pair,
                                                 int tile, const float* bp, int dk) {
#pragma unroll
  for (int i = 0; i < 4 * NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) z[i][c] = make_float2(0.f, 0.f);
  float4 u[2 * NT], b[4], un[2 * NT], bn[4];
  auto load = [&](int d, float4(&x)[2 * NT], float4(&q)[4]) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      x[2 * t] = lds4(xp + t * tile + 2 * d);
      x[2 * t + 1] = lds4(xp + t * tile + pair + 2 * d);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = lds4(bp + (d + (j >> 1)) * kF32CT + (j & 1) * 64);
  };
  load(0, u, b);
#pragma unroll 2
  for (int d = 0; d < dk; d += 2) {
    load(d + 2 < dk ? d + 2 : d, un, bn);
#pragma unroll
    for (int k = 0; k < 2 * NT; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) {      // row 2 k + h of this thread's
        const float xa = h ? u[k].y : u[k].x, xb = h ? u[k].w : u[k].z;
        float2(&zr)[4] = z[2 * k + h];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          zr[2 * j] = __ffma2_rn(make_float2(xa, xa), make_float2(b[j].x, b[j].y), zr[2 * j]);
          zr[2 * j + 1] =
              __ffma2_rn(make_float2(xa, xa), make_float2(b[j].z, b[j].w), zr[2 * j + 1]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          zr[2 * j] =
              __ffma2_rn(make_float2(xb, xb), make_float2(b[2 + j].x, b[2 + j].y), zr[2 * j]);
          zr[2 * j + 1] = __ffma2_rn(make_float2(xb, xb), make_float2(b[2 + j].z, b[2 + j].w),
                                     zr[2 * j + 1]);
        }
      }
#pragma unroll
    for (int k = 0; k < 2 * NT; ++k) u[k] = un[k];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = bn[j];
  }
}

// Epilogue of one thread: adds its rows' -(|z|/2 + ln(1 + e^-|z|)) to each
// chain's Kahan sum and passes R of row i to `store`.
template <class Store>
__device__ __forceinline__ void f32_epilogue(const float (&z)[4][8], const float (&yr)[4],
                                             int nvalid, float (&lsum)[8], float (&lcomp)[8],
                                             Store&& store) {
  float sabs[8], prod[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) { sabs[c] = 0.f; prod[c] = 1.f; }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float r[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) f32_residual(z[i][c], yr[i], i < nvalid, sabs[c], prod[c], r[c]);
    store(i, r);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) kahan_add(f32_like(sabs[c], prod[c]), lsum[c], lcomp[c]);
}

// The epilogue of four rows x four pairs of chains; `store` gets R of a row.
template <class Store>
__device__ __forceinline__ void f32_epilogue_pairs(const float2 (&z)[8][4], int first,
                                                   const float (&yr)[4], int nvalid,
                                                   float (&lsum)[8], float (&lcomp)[8],
                                                   Store&& store) {
  float2 sabs[4], prod[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    sabs[c] = make_float2(0.f, 0.f);
    prod[c] = make_float2(1.f, 1.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 r[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      r[c] = f32_residual2(z[first + i][c], yr[i], i < nvalid, sabs[c], prod[c]);
    store(i, r);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    kahan_add(f32_like(sabs[c].x, prod[c].x), lsum[2 * c], lcomp[2 * c]);
    kahan_add(f32_like(sabs[c].y, prod[c].y), lsum[2 * c + 1], lcomp[2 * c + 1]);
  }
}

template <int KD>
__global__ void __launch_bounds__(kF32Threads, 1)
logreg_f32_kernel(const float* __restrict__ X2, const float* __restrict__ ym, int N, int D,
                  const float* __restrict__ Q, int ldq, const int* __restrict__ n_dev,
                  int c_base, int c_lim, int grid, double* __restrict__ lpart,
                  float* __restrict__ gpart, int* __restrict__ err) {
  using L = F32Layout<KD>;
  constexpr int Dp = L::kDp;
  extern __shared__ __align__(128) unsigned char smem[];
  const int n = chunk_count(*n_dev, c_base, c_lim);
  const int row_tiles = (N + kF32RT - 1) / kF32RT;
  const int S = f32_splits(n, grid, row_tiles);
  const int tiles = (n + kF32CT - 1) / kF32CT;
  if (S == 0 || (int)blockIdx.x >= tiles * S) return;
  const int tile = blockIdx.x % tiles, split = blockIdx.x / tiles;
  const int c0 = tile * kF32CT;
  const int rt_begin = (int)((long long)split * row_tiles / S);
  const int rt_end = (int)((long long)(split + 1) * row_tiles / S);
  const int T = rt_end - rt_begin;

  float* Bt = reinterpret_cast<float*>(smem + L::kBt);
  float* Xs = reinterpret_cast<float*>(smem + L::kX);
  float* Ys = reinterpret_cast<float*>(smem + L::kY);
  float* Rs = reinterpret_cast<float*>(smem + L::kR);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBar);
  const int tid = threadIdx.x;

  int issued = 0;              // thread 0: row tiles whose copies were issued
  auto issue = [&](int it) {   // thread 0: bulk copies of row tile rt_begin + it
    const int st = it & 1;
    issued = it + 1;
    const size_t r0 = (size_t)(rt_begin + it) * kF32RT;
    tc::fence_proxy_async_smem();
    tc::mbar_arrive_expect_tx(&full[st], (uint32_t)(L::kXStage + kF32RT * 4));
    tc::bulk_load(Xs + st * (L::kXStage / 4), X2 + r0 * Dp, (uint32_t)L::kXStage, &full[st]);
    tc::bulk_load(Ys + st * kF32RT, ym + r0, (uint32_t)(kF32RT * 4), &full[st]);
  };
  if (tid == 0) {
    tc::mbar_init(&full[0], 1);
    tc::mbar_init(&full[1], 1);
    tc::fence_mbar_init();
    if (T > 0) issue(0);
    if (T > 1) issue(1);
  }
  // Chain states, transposed: Bt[d][c] = Q[c0 + c][d], zero outside (n, D).
  for (int i = tid; i < Dp * kF32CT; i += kF32Threads) {
    const int c = i / Dp, d = i - c * Dp;
    Bt[d * kF32CT + c] = (c0 + c < n && d < D) ? Q[(size_t)(c0 + c) * ldq + d] : 0.f;
  }
  __syncthreads();

  const int ty = tid >> 4, tx = tid & 15;   // phase 1: rows 4 ty.., chains 4 tx.., 64 + 4 tx..
  const int cg = ty, fg = tx;               // phase 2: chains 4 cg.., 64 + 4 cg..; f = fg + 16 j
  const int dk = (D + 1) & ~1;              // K extent of phase 1 (B^T rows >= D are zero)
  float g[8][KD];
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int j = 0; j < KD; ++j) g[c][j] = 0.f;
  // Per chain: Kahan sum over tiles of -(sum |z|/2 + sum ln(1 + e^-|z|)).
  float lsum[8], lcomp[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) lsum[c] = lcomp[c] = 0.f;
  bool ok = true;        // this thread's waits succeeded
  bool failed = false;   // some thread's wait ran out (uniform across the CTA)
  int it = 0;

  for (; it < T; ++it) {
    const int st = it & 1;
    if (!tc::mbar_wait(&full[st], (uint32_t)(it >> 1) & 1, kF32WaitNs)) ok = false;
    const float* xs = Xs + st * (L::kXStage / 4);
    // ---- phase 1: Z = X_tile B^T ----
    float z[4][8];
    f32_phase1(z, xs + (2 * ty) * Dp * 2, Dp * 2, Bt + 4 * tx, dk);
    // ---- epilogue: log-likelihood sums and R ----
    const float4 yv = lds4(Ys + st * kF32RT + 4 * ty);
    const float yr[4] = {yv.x, yv.y, yv.z, yv.w};
    const int nvalid = N - (rt_begin + it) * kF32RT - 4 * ty;   // rows of mine that exist
    f32_epilogue(z, yr, nvalid, lsum, lcomp, [&](int i, const float(&r)[8]) {
      float* rrow = Rs + (4 * ty + i) * kF32CT;
      *reinterpret_cast<float4*>(rrow + 4 * tx) = make_float4(r[0], r[1], r[2], r[3]);
      *reinterpret_cast<float4*>(rrow + 64 + 4 * tx) = make_float4(r[4], r[5], r[6], r[7]);
    });
    if (__syncthreads_or(!ok)) {   // R complete (and every thread's wait succeeded)
      failed = true;
      break;
    }
    // ---- phase 2: G += R^T X_tile ----
    // Register double buffering of the residual rows and the row pair of X,
    // as in phase 1.
    const float* rp = Rs + 4 * cg;
    const float* xq = xs + 2 * fg;
    float4 ra0 = lds4(rp), ra1 = lds4(rp + 64), rb0 = lds4(rp + kF32CT),
           rb1 = lds4(rp + kF32CT + 64);
    float2 xv[KD];
#pragma unroll
    for (int j = 0; j < KD; ++j) xv[j] = *reinterpret_cast<const float2*>(xq + 32 * j);
#pragma unroll 2
    for (int p = 0; p < kF32RT / 2; ++p) {
      const int pn = p + 1 < kF32RT / 2 ? p + 1 : p;
      const float* rn = rp + (2 * pn) * kF32CT;
      const float4 ra0n = lds4(rn), ra1n = lds4(rn + 64), rb0n = lds4(rn + kF32CT),
                   rb1n = lds4(rn + kF32CT + 64);
      float2 xvn[KD];
#pragma unroll
      for (int j = 0; j < KD; ++j)
        xvn[j] = *reinterpret_cast<const float2*>(xq + pn * Dp * 2 + 32 * j);
      const float r0[8] = {ra0.x, ra0.y, ra0.z, ra0.w, ra1.x, ra1.y, ra1.z, ra1.w};
      const float r1[8] = {rb0.x, rb0.y, rb0.z, rb0.w, rb1.x, rb1.y, rb1.z, rb1.w};
#pragma unroll
      for (int j = 0; j < KD; ++j)
#pragma unroll
        for (int c = 0; c < 8; ++c)
          g[c][j] = fmaf(r1[c], xv[j].y, fmaf(r0[c], xv[j].x, g[c][j]));
      ra0 = ra0n; ra1 = ra1n; rb0 = rb0n; rb1 = rb1n;
#pragma unroll
      for (int j = 0; j < KD; ++j) xv[j] = xvn[j];
    }
    __syncthreads();   // stage st and R are free
    if (tid == 0 && it + 2 < T) issue(it + 2);
  }

  if (failed) {
    if (tid == 0) {
      tc::record_error(err, kF32TimeoutCode);
      // Let copies still in flight (tiles it .. issued - 1) land before the
      // CTA exits; each wait is bounded.
      for (int j = it; j < issued; ++j)
        tc::mbar_wait(&full[j & 1], (uint32_t)(j >> 1) & 1, kF32WaitNs);
    }
    return;
  }
  // Per-chain log-likelihood partial: sum the 16 row groups in fixed order.
  double* red = reinterpret_cast<double*>(Rs);     // [16][128]
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int cc = c < 4 ? 4 * tx + c : 64 + 4 * tx + (c - 4);
    red[ty * kF32CT + cc] = (double)lsum[c] - (double)lcomp[c];
  }
  __syncthreads();
  if (tid < kF32CT && c0 + tid < n) {
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < 16; ++t) s += red[t * kF32CT + tid];
    lpart[(size_t)split * n + c0 + tid] = s;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int cc = c0 + (c < 4 ? 4 * cg + c : 64 + 4 * cg + (c - 4));
    if (cc >= n) continue;
    float* dst = gpart + ((size_t)split * n + cc) * D;
#pragma unroll
    for (int j = 0; j < KD; ++j) {
      const int d = fg + 16 * j;
      if (d < D) dst[d] = g[c][j];
    }
  }
}

// ---------------------------------------------------------------------------
// Phase 2 on the tensor cores (see the head of this file).
//
// Two groups of four warps, a warp of each on every SM quarter, take the upper
// and the lower 32 rows of each tile, and have their own stages, accumulators
// and a service warp that loads their rows and issues their MMAs.  A group runs
// phase 1 over the rows of two tiles (8 rows x 8 chains a thread), then the two
// epilogues, while its next rows load and its MMAs (6 a tile) run.  Group 1
// begins with a single tile, so that the groups are half a turn apart and one's
// epilogue (MUFU and issue) fills what the other's phase 1 (FMA pipe) leaves.
//
// What bounds it: the FMA pipe in phase 1, half of the kernel (107 of 128 FMAs a
// clock and SM), and the issue of the epilogues.  An evaluation at 1e5 rows, 1024
// chains: 516 us at 100 features (both phases on the CUDA cores: 849; this
// kernel with one group of eight warps, epilogues together: 547), 221 at 25
// (344), 54 at 4 and 256 chains (72).
// ---------------------------------------------------------------------------
constexpr int kF32TcThreads = kF32Threads + 64;
constexpr int kHalf = kF32RT / 2;           // rows of a tile in each group
constexpr int kRBox = kHalf * 128;          // [32 rows][128 B]: 64 chains
constexpr int kXBox = 2 * kRBox;            // [2 tiles][32 rows][128 B]: 64 features

template <int KD>
struct F32TcLayout {
  static constexpr int kDp = 16 * KD;
  static constexpr int kNkb = (KD + 3) / 4;                  // 64-feature blocks
  static constexpr int kGCols = KD <= 2 ? 32 : KD <= 4 ? 64 : 128;
  static constexpr int kX16Group = 2 * kNkb * kXBox;         // hi, lo
  static constexpr int kR16Group = 4 * kRBox;                // hi, lo of 2 x 64 chains
  static constexpr int kXHalf = kHalf * kDp * 4;             // X2 of a tile's rows of a group
  static constexpr int kX16 = 0;                              // [group]
  static constexpr int kR16 = kX16 + 2 * kX16Group;           // [group]
  static constexpr int kBt = kR16 + 2 * kR16Group;            // [Dp][128] float
  static constexpr int kX = kBt + kDp * kF32CT * 4;           // [group][2 tiles]
  static constexpr int kY = kX + 4 * kXHalf;                  // [group][2 tiles][32] float
  static constexpr int kCtl = kY + 2 * kF32RT * 4;
  static constexpr int kBytes = kCtl + 256 + 1024;
  // After the loop: log-likelihood sums over R, the gradient tile over B^T and X2.
  static_assert(16 * kF32CT * 8 <= 2 * kR16Group, "reduction scratch fits R");
  static_assert(kF32CT * (kDp + 1) * 4 <= kY - kBt, "gradient tile fits B^T and X2");
  static_assert(kBytes <= 232448, "shared memory over the sm_103a limit");
};

struct F32TcBars {
  struct Group {
    uint64_t x_full, x_free, x16_full, r_full, mma_done;
  } group[2];
};

// Tiles of turn j of a group: [first, first + count).
__device__ __forceinline__ int turn_first(int group, int j) {
  return group == 0 || j == 0 ? 2 * j : 2 * j - 1;
}
__device__ __forceinline__ int turn_count(int group, int j, int T) {
  const int left = T - turn_first(group, j);
  const int most = group == 1 && j == 0 ? 1 : 2;
  return left < most ? left : most;
}

template <int KD>
__global__ void __launch_bounds__(kF32TcThreads, 1)
logreg_f32_tc_kernel(const __grid_constant__ CUtensorMap himap,
                     const __grid_constant__ CUtensorMap lomap, const float* __restrict__ X2,
                     const float* __restrict__ ym, const float* __restrict__ gscale, int N, int D,
                     const float* __restrict__ Q, int ldq, const int* __restrict__ n_dev,
                     int c_base, int c_lim, int grid, double* __restrict__ lpart,
                     float* __restrict__ gpart, int* __restrict__ err) {
  using L = F32TcLayout<KD>;
  constexpr int Dp = L::kDp;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int n = chunk_count(*n_dev, c_base, c_lim);
  const int row_tiles = (N + kF32RT - 1) / kF32RT;
  const int S = f32_splits(n, grid, row_tiles);
  const int tiles = (n + kF32CT - 1) / kF32CT;
  if (S == 0 || (int)blockIdx.x >= tiles * S) return;
  const int tile = blockIdx.x % tiles, split = blockIdx.x / tiles;
  const int c0 = tile * kF32CT;
  const int rt_begin = (int)((long long)split * row_tiles / S);
  const int rt_end = (int)((long long)(split + 1) * row_tiles / S);
  const int T = rt_end - rt_begin;

  float* Bt = reinterpret_cast<float*>(smem + L::kBt);
  F32TcBars* all = reinterpret_cast<F32TcBars*>(smem + L::kCtl);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kCtl + sizeof(F32TcBars));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = warp < 8 ? warp >> 2 : warp - 8;
  F32TcBars::Group* bars = &all->group[group];
  unsigned char* X16 = smem + L::kX16 + group * L::kX16Group;
  unsigned char* R16 = smem + L::kR16 + group * L::kR16Group;
  float* Xs = reinterpret_cast<float*>(smem + L::kX + group * 2 * L::kXHalf);
  float* Ys = reinterpret_cast<float*>(smem + L::kY) + group * kF32RT;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      F32TcBars::Group& b = all->group[i];
      tc::mbar_init(&b.x_full, 1);
      tc::mbar_init(&b.x_free, 4);
      tc::mbar_init(&b.x16_full, 1);
      tc::mbar_init(&b.r_full, 4);
      tc::mbar_init(&b.mma_done, 1);
    }
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  // TMEM: G of a group's turn (two groups), then the groups' sums.
  if (warp == 8) tc::tmem_alloc(tmem_slot, 4 * L::kGCols);
  // Chain states, transposed: Bt[d][c] = Q[c0 + c][d], zero outside (n, D).
  // Lanes run over chains: conflict-free stores, and a row of Q stays in L1.
  for (int i = tid; i < Dp * kF32CT; i += kF32TcThreads) {
    const int c = i & (kF32CT - 1), d = i / kF32CT;
    Bt[i] = (c0 + c < n && d < D) ? Q[(size_t)(c0 + c) * ldq + d] : 0.f;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tg = tmem + group * L::kGCols, tsum = tmem + (2 + group) * L::kGCols;

  if (warp >= 8) {
    // ---------------- a group's loads and MMAs ----------------
    if (tc::elect_one()) {
      // A turn's rows: 32 of each tile, X2 and y, and the FP16 form.
      auto load_x = [&](int j) {
        const int first = turn_first(group, j), count = turn_count(group, j, T);
        tc::mbar_arrive_expect_tx(&bars->x_full, (uint32_t)(count * (L::kXHalf + kHalf * 4)));
        for (int t = 0; t < count; ++t) {
          const size_t r0 = (size_t)(rt_begin + first + t) * kF32RT + group * kHalf;
          tc::bulk_load(Xs + t * (L::kXHalf / 4), X2 + r0 * Dp, (uint32_t)L::kXHalf, &bars->x_full);
          tc::bulk_load(Ys + t * kHalf, ym + r0, (uint32_t)(kHalf * 4), &bars->x_full);
        }
      };
      auto load_x16 = [&](int j) {
        const int first = turn_first(group, j), count = turn_count(group, j, T);
        tc::mbar_arrive_expect_tx(&bars->x16_full, (uint32_t)(count * 2 * L::kNkb * kRBox));
        for (int t = 0; t < count; ++t) {
          const int r0 = (rt_begin + first + t) * kF32RT + group * kHalf;
#pragma unroll
          for (int kb = 0; kb < L::kNkb; ++kb) {
            tc::tma_load_2d(X16 + kb * kXBox + t * kRBox, &himap, kb * 64, r0, &bars->x16_full);
            tc::tma_load_2d(X16 + (L::kNkb + kb) * kXBox + t * kRBox, &lomap, kb * 64, r0,
                            &bars->x16_full);
          }
        }
      };
      if (T > 0) {
        load_x(0);
        load_x16(0);
      }
      int nx = T > 0, nx16 = nx;      // turns whose loads were issued
      constexpr uint32_t idesc = tc::idesc_16bit_f32(128, Dp, true, true, false);
      const uint64_t rd = tc::smem_desc_sw128(tc::smem_u32(R16), kRBox, 1024);
      const uint64_t xd = tc::smem_desc_sw128(tc::smem_u32(X16), kXBox, 1024);
      constexpr uint64_t kRlo = 2 * kRBox >> 4, kXlo = L::kNkb * kXBox >> 4;
      bool ok = true;
      int it = 0;
      for (int j = 0; ok && turn_first(group, j) < T; ++j) {
        const int count = turn_count(group, j, T);
        const bool more = turn_first(group, j + 1) < T;
        // Phase 1 of the turn is done: the next rows load during its epilogue.
        if (more) {
          ok = wait_or_abort(&bars->x_free, (uint32_t)j & 1, abort_flag);
          if (!ok) break;
          load_x(nx++);
        }
        ok = wait_or_abort(&bars->x16_full, (uint32_t)j & 1, abort_flag);
        for (int t = 0; ok && t < count; ++t, ++it) {
          ok = wait_or_abort(&bars->r_full, (uint32_t)it & 1, abort_flag);
          if (!ok) break;
          tc::tc_fence_after();
          const uint64_t xt = xd + (uint64_t)((t * kRBox) >> 4);
#pragma unroll
          for (int ks = 0; ks < kHalf / 16; ++ks) {
            const uint64_t o = (uint64_t)((ks * 2048) >> 4);
            tc::mma_16bit(tg, rd + kRlo + o, xt + o, idesc, t > 0 || ks > 0 ? 1u : 0u);
            tc::mma_16bit(tg, rd + o, xt + kXlo + o, idesc, 1u);
          }
#pragma unroll
          for (int ks = 0; ks < kHalf / 16; ++ks) {
            const uint64_t o = (uint64_t)((ks * 2048) >> 4);
            tc::mma_16bit(tg, rd + o, xt + o, idesc, 1u);
          }
          tc::mma_commit(&bars->mma_done);
        }
        if (ok && more) {
          ok = wait_or_abort(&bars->mma_done, (uint32_t)(it - 1) & 1, abort_flag);
          if (ok) load_x16(nx16++);
        }
      }
      if (!ok) {
        tc::record_error(err, kF32TimeoutCode);
        *abort_flag = 1;
        // Let the MMAs and the copies still in flight end before the CTA exits.
        if (it > 0) tc::mbar_wait(&bars->mma_done, (uint32_t)(it - 1) & 1, kWaitLimitNs);
        if (nx > 0) tc::mbar_wait(&bars->x_full, (uint32_t)(nx - 1) & 1, kWaitLimitNs);
        if (nx16 > 0) tc::mbar_wait(&bars->x16_full, (uint32_t)(nx16 - 1) & 1, kWaitLimitNs);
      }
    }
    __syncwarp();
  } else {
    const int ty = tid >> 4, tx = tid & 15;   // rows 4 ty.., chains 4 tx.., 64 + 4 tx..
    const int gy = ty & 7;                    // ty within the group
    const int dk = (D + 1) & ~1;              // K extent of phase 1 (B^T rows >= D are zero)
    const uint32_t quarter = (uint32_t)((warp & 3) * 32) << 16;
    // Per chain: Kahan sum over tiles of -(sum |z|/2 + sum ln(1 + e^-|z|)).
    float lsum[8], lcomp[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) lsum[c] = lcomp[c] = 0.f;
    bool ok = true, summed = false;
    // Adds G of a turn to the sum of the turns before, which is kept in TMEM
    // beside it: the registers for it would not be left.
    auto drain = [&]() {
      tc::tc_fence_after();
#pragma unroll
      for (int j = 0; j < 2 * KD; ++j) {
        float v[8], sum[8];
        tc::tmem_ld8(tg + quarter + 8 * j, v);
        if (summed) tc::tmem_ld8(tsum + quarter + 8 * j, sum);
        tc::tmem_ld_wait();
        if (summed) {
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] += sum[e];
        }
        tc::tmem_st8(tsum + quarter + 8 * j, v);
      }
      tc::tmem_st_wait();
      tc::tc_fence_before();
      summed = true;
    };
    for (int j = 0; turn_first(group, j) < T && ok; ++j) {
      const int first = turn_first(group, j), count = turn_count(group, j, T);
      if (!warp_wait(&bars->x_full, (uint32_t)j & 1, abort_flag)) {
        ok = false;
        break;
      }
      // ---- phase 1: Z = X_tile B^T of the turn's tiles ----
      float2 z[8][4];
      const float* xp = Xs + (2 * gy) * Dp * 2;
      if (count == 2)
        f32_phase1_pairs<2>(z, xp, Dp * 2, L::kXHalf / 4, Bt + 4 * tx, dk);
      else
        f32_phase1_pairs<1>(z, xp, Dp * 2, L::kXHalf / 4, Bt + 4 * tx, dk);
      float4 yv[2];
      yv[0] = lds4(Ys + 4 * gy);
      yv[1] = lds4(Ys + kHalf + 4 * gy);
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars->x_free);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int it = first + t;
        if (t == 1 && count == 1) break;
        // The MMAs of the tile before are done: R is free, and with a new turn
        // G of the last one is complete.
        if (it > 0) {
          if (!warp_wait(&bars->mma_done, (uint32_t)(it - 1) & 1, abort_flag)) {
            ok = false;
            break;
          }
          if (t == 0) drain();
        }
        // ---- epilogue: log-likelihood sums, R' in FP16 hi + lo ----
        const float yr[4] = {yv[t].x, yv[t].y, yv[t].z, yv[t].w};
        const int nvalid = N - (rt_begin + it) * kF32RT - 4 * ty;   // rows of mine that exist
        auto put = [&](int i, const float2(&r)[4]) {
          const uint32_t off = tc::sw128_offset(4 * gy + i, 4 * tx);
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            uint32_t hi[2], lo[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float2 v = __fmul2_rn(r[2 * b + e], make_float2(kF16Scale, kF16Scale));
              const __half2 h = __float22half2_rn(v);
              const float2 hf = __half22float2(h);
              const __half2 l =
                  __float22half2_rn(__fadd2_rn(v, make_float2(-hf.x, -hf.y)));
              hi[e] = *reinterpret_cast<const uint32_t*>(&h);
              lo[e] = *reinterpret_cast<const uint32_t*>(&l);
            }
            *reinterpret_cast<uint2*>(R16 + b * kRBox + off) = make_uint2(hi[0], hi[1]);
            *reinterpret_cast<uint2*>(R16 + (2 + b) * kRBox + off) = make_uint2(lo[0], lo[1]);
          }
        };
        f32_epilogue_pairs(z, 4 * t, yr, nvalid, lsum, lcomp, put);
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bars->r_full);
      }
    }
    if (ok && T > 0) {
      ok = warp_wait(&bars->mma_done, (uint32_t)(T - 1) & 1, abort_flag);
      if (ok) drain();
    }
    if (!ok) {
      tc::record_error(err, kF32TimeoutCode);
      *abort_flag = 1;
    }
    // Every warp is past its last read of B^T, X2 and R (or has given up), and
    // both groups' sums are complete.
    named_barrier(1, kF32Threads);
    const bool good = *abort_flag == 0;
    if (good) {
      tc::tc_fence_after();
      double* red = reinterpret_cast<double*>(smem + L::kR16);    // [16][128]
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int cc = c < 4 ? 4 * tx + c : 64 + 4 * tx + (c - 4);
        red[ty * kF32CT + cc] = (double)lsum[c] - (double)lcomp[c];
      }
      // This group's half of the features of its lanes' chains.
      const int gc = (warp & 3) * 32 + lane, gf = group * 8 * KD;
#pragma unroll
      for (int j = 0; j < KD; ++j) {
        float v0[8], v1[8];
        tc::tmem_ld8(tmem + 2 * L::kGCols + quarter + gf + 8 * j, v0);
        tc::tmem_ld8(tmem + 3 * L::kGCols + quarter + gf + 8 * j, v1);
        tc::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) Bt[gc * (Dp + 1) + gf + 8 * j + e] = v0[e] + v1[e];
      }
    }
    named_barrier(1, kF32Threads);
    if (good) {
      const double* red = reinterpret_cast<const double*>(smem + L::kR16);
      if (tid < kF32CT && c0 + tid < n) {
        double s = 0.0;
#pragma unroll
        for (int t = 0; t < 16; ++t) s += red[t * kF32CT + tid];
        lpart[(size_t)split * n + c0 + tid] = s;
      }
      for (int cc = warp; cc < kF32CT; cc += kF32Threads / 32) {
        if (c0 + cc >= n) break;
        float* dst = gpart + ((size_t)split * n + c0 + cc) * D;
        for (int d = lane; d < D; d += 32) dst[d] = Bt[cc * (Dp + 1) + d] * gscale[d];
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 4 * L::kGCols);
  }
}

// X [N][D] -> X2 [N2/2][Dp][2] (row pairs, zero padding) and ym = y - 1/2
// (zero past N), N2 = N rounded up to whole row tiles.
__global__ void f32_pack_kernel(const float* __restrict__ X, const float* __restrict__ y,
                                int64_t N, int D, int Dp, int64_t N2, float* __restrict__ X2,
                                float* __restrict__ ym) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N2) ym[i] = i < N ? y[i] - 0.5f : 0.f;
  if (i >= N2 * Dp) return;
  const int64_t r = i / Dp;
  const int d = (int)(i - r * Dp);
  X2[((r >> 1) * Dp + d) * 2 + (r & 1)] = (r < N && d < D) ? X[r * D + d] : 0.f;
}

// lin[d] = sum_r (y_r - 1/2) X[r][d] in float64 and a fixed order: block b
// sums rows [b chunk, (b + 1) chunk) into part[b][d]; blocks added in order.
__global__ void f32_lin_partial(const float* __restrict__ X, const float* __restrict__ y,
                                int64_t N, int D, int64_t chunk, double* __restrict__ part) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk;
  const int64_t r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    double acc = 0.0;
#pragma unroll 8
    for (int64_t r = r0; r < r1; ++r) acc += ((double)y[r] - 0.5) * (double)X[r * D + d];
    part[(size_t)blockIdx.x * D + d] = acc;
  }
}

__global__ void f32_lin_sum(const double* __restrict__ part, int nb, int D,
                            double* __restrict__ lin) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  double acc = 0.0;
  for (int b = 0; b < nb; ++b) acc += part[(size_t)b * D + d];
  lin[d] = acc;
}

template <int KD>
void f32_set_smem() {
  GBM_CUDA(cudaFuncSetAttribute(logreg_f32_kernel<KD>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                F32Layout<KD>::kBytes));
  GBM_CUDA(cudaFuncSetAttribute(logreg_f32_tc_kernel<KD>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                F32TcLayout<KD>::kBytes));
}

// From kPairRows rows on phase 2 runs on the tensor cores.  It is the faster one from
// there on: 4096 rows x 10 features x 64 chains 26.2 us an evaluation (27.7 on
// the CUDA cores), x 100 30.1 (35.2), 8192 x 4 x 1024 31.3 (35.0).  Below, where
// an evaluation is launch latency for the most part (2000 x 100 x 64: 36
// against 43 us), the gradient keeps its FP32 summation order: a sampler run
// over a small data set repeats to the digit.

class LogregF32 final : public Target {
 public:
  LogregF32(gbm_context* ctx, const float* X, int64_t n, int64_t d, const float* y,
            float prior_scale, bool pairs)
      : N_(n), D_(d) {
    dim = d;
    kd_ = width(d);
    dp_ = 16 * kd_;
    n2_ = (n + kF32RT - 1) / kF32RT * kF32RT;
    x2_.reserve(sizeof(float) * (size_t)n2_ * dp_);
    ym_.reserve(sizeof(float) * (size_t)n2_);
    const int64_t total = n2_ * dp_;
    f32_pack_kernel<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(
        X, y, N_, (int)D_, dp_, n2_, x2_.as<float>(), ym_.as<float>());
    GBM_CUDA(cudaGetLastError());
    {
      const int nb = 2 * ctx->num_sms;
      const int64_t chunk = (N_ + nb - 1) / nb;
      DeviceBuffer part;
      part.reserve(sizeof(double) * (size_t)nb * D_);
      lin_.reserve(sizeof(double) * (size_t)D_);
      f32_lin_partial<<<nb, 128, 0, ctx->stream>>>(X, y, N_, (int)D_, chunk,
                                                   part.as<double>());
      f32_lin_sum<<<(unsigned)((D_ + 127) / 128), 128, 0, ctx->stream>>>(
          part.as<double>(), nb, (int)D_, lin_.as<double>());
      GBM_CUDA(cudaGetLastError());
      GBM_CUDA(cudaStreamSynchronize(ctx->stream));   // `part` is freed on scope exit
    }
    inv_var_ = 1.f / (prior_scale * prior_scale);
    log_norm_ = -log((double)prior_scale) - 0.5 * log(2.0 * M_PI);
    grid_ = ctx->num_sms;
    err_dev_ = ctx->err_dev;
    tc_ = pairs && n >= kPairRows && x16_.prepare(ctx, X, ym_.as<float>(), N_, (int)D_, dp_, kHalf);
    switch (kd_) {
      case 1: f32_set_smem<1>(); break;
      case 2: f32_set_smem<2>(); break;
      case 3: f32_set_smem<3>(); break;
      case 4: f32_set_smem<4>(); break;
      case 6: f32_set_smem<6>(); break;
      case 7: f32_set_smem<7>(); break;
      default: f32_set_smem<8>(); break;
    }
    if (!tc_) {
      prepare_leapfrogs<1>();
      prepare_leapfrogs<2>();
      prepare_leapfrogs<4>();
    }
  }

  static int width(int64_t d) {      // in 16 features
    const int kd = (int)((d + 15) / 16);
    return kd == 5 ? 6 : kd;   // instantiated widths: 1 2 3 4 6 7 8
  }
  static size_t work_bytes(int grid, int64_t cap, int64_t d) {
    const size_t rows = (size_t)grid * kF32CT + (size_t)cap;
    return rows * sizeof(double) + rows * (size_t)d * sizeof(float) + 256;
  }
  size_t workspace_bytes(int64_t cap) const override { return work_bytes(grid_, cap, D_); }

  // One launch covers at most grid_ * 128 chains (one work item per CTA);
  // larger batches run as consecutive chunks that share the workspace.
  void eval(const float* q, int ldq, const int* n_dev, int cap, double* logp, float* grad,
            int ldg, void* ws, cudaStream_t s) override {
    const size_t rows = (size_t)grid_ * kF32CT + (size_t)cap;
    double* lpart = static_cast<double*>(ws);
    float* gpart = reinterpret_cast<float*>(lpart + rows);
    const int N = (int)N_, D = (int)D_;
    const int lim = grid_ * kF32CT;
    for (int base = 0; base < cap; base += lim) {
      const float* qc = q + (size_t)base * ldq;
      const int g = work_grid(grid_, std::min(lim, cap - base), kF32CT, N_, kMinSplitRows);
#define GBM_F32_LAUNCH(KD_)                                                                \
  if (tc_)                                                                                 \
    logreg_f32_tc_kernel<KD_><<<g, kF32TcThreads, F32TcLayout<KD_>::kBytes, s>>>(             \
        x16_.hi, x16_.lo, x2_.as<float>(), ym_.as<float>(), x16_.gscale, N, D, qc, ldq,\
        n_dev, base, lim, g, lpart, gpart, err_dev_);                                        \
  else                                                                                     \
    logreg_f32_kernel<KD_><<<g, kF32Threads, F32Layout<KD_>::kBytes, s>>>(                    \
        x2_.as<float>(), ym_.as<float>(), N, D, qc, ldq, n_dev, base, lim, g, lpart, gpart,    \
        err_dev_)
      switch (kd_) {
        case 1: GBM_F32_LAUNCH(1); break;
        case 2: GBM_F32_LAUNCH(2); break;
        case 3: GBM_F32_LAUNCH(3); break;
        case 4: GBM_F32_LAUNCH(4); break;
        case 6: GBM_F32_LAUNCH(6); break;
        case 7: GBM_F32_LAUNCH(7); break;
        default: GBM_F32_LAUNCH(8); break;
      }
#undef GBM_F32_LAUNCH
      GBM_CUDA(cudaGetLastError());
      launch_split_reduce(lpart, gpart, qc, ldq, n_dev, base, lim, std::min(lim, cap - base),
                          kF32CT, kF32RT, g, N, D, inv_var_, log_norm_, lin_.as<double>(),
                          logp + base, grad + (size_t)base * ldg, ldg, s);
    }
  }

  // A trajectory of logreg_f32_kernel's gradients in one launch, while X and the
  // chains fit the GPU's shared memory.
  bool leapfrogs(float* q, float* p, float* g, double* logp, int ld, int chains, const float* eps,
                 int per_chain, int steps, cudaStream_t s) override {
    LeapShape h;
    if (tc_ || !leap_shape(N_, (int)D_, chains, grid_, kF32CT, &h)) return false;
    auto go = [&](auto launch) {
      launch(h, x2_.as<float>(), ym_.as<float>(), (int)N_, dp_, chains, steps, eps, per_chain,
             inv_var_, log_norm_, lin_.as<double>(), q, p, g, logp, ld, s);
    };
    if (h.G == 1)
      go(launch_leapfrogs<1>);
    else if (h.G == 2)
      go(launch_leapfrogs<2>);
    else
      go(launch_leapfrogs<4>);
    return true;
  }

  int launches_per_eval(int64_t cap) const override {
    return 2 * (int)((cap + (int64_t)grid_ * kF32CT - 1) / ((int64_t)grid_ * kF32CT));
  }
  double flops(int64_t n) const override { return 4.0 * (double)N_ * D_ * n; }
  double bytes(int64_t n) const override {
    return 4.0 * (double)N_ * D_ + 4.0 * N_ + 8.0 * (double)n * D_ + 8.0 * n;
  }

 private:
  int64_t N_, D_, n2_ = 0;
  int kd_ = 1, dp_ = 16, grid_ = 0;
  float inv_var_ = 1.f;
  double log_norm_ = 0.0;
  int* err_dev_ = nullptr;
  DeviceBuffer x2_, ym_, lin_;
  bool tc_ = false;            // phase 2 on the tensor cores
  F16Rows x16_;
};

}  // namespace

std::unique_ptr<Target> make_logreg_f32(gbm_context* ctx, const float* X, int64_t n, int64_t d,
                                        const float* y, float prior_scale, bool pairs) {
  if (d > 128) return nullptr;
  return std::unique_ptr<Target>(new LogregF32(ctx, X, n, d, y, prior_scale, pairs));
}

size_t logreg_f32_bytes(int64_t n, int64_t d, int64_t chains, int num_sms, bool pairs) {
  const int dp = 16 * LogregF32::width(d);
  const size_t n2 = (size_t)((n + kF32RT - 1) / kF32RT * kF32RT);
  return 4 * n2 * (dp + 1) + 8 * (size_t)d * (2 * num_sms + 1) +
         (pairs && n >= kPairRows ? F16Rows::bytes(n, (int)d, dp, num_sms) : 0) +
         LogregF32::work_bytes(num_sms, chains, d);
}

}  // namespace gbm
