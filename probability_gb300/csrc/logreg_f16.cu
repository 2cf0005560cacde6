// The FP32 logistic-regression target for up to 128 features on the tensor
// cores: log-density and gradient with the accuracy of FP32 arithmetic, from
// FP16 operands.
//
// Mathematics as in logreg_f32.cu.  Per 64-row tile of X and 128 chains,
//   Z^T  = B X_tile^T                 (M = 128 chains, N = 64 rows)
//   R^T  = (y - sigmoid(Z))^T         (epilogue)
//   G^T += R^T X_tile                 (M = 128 chains, N = features, K = 64 rows)
//
// Splits.  Features, chain states and residuals are scaled by powers of two
// and cut into FP16 slices, leading digits first:
//   X' = X1 + X2 + X3   X1 of 6 bits on the feature's own scale, X2 and X3 the
//                       remainders: X' to 2^-31 of the feature's largest;
//   B' = B1 + B2 + B3   B1 of 11 bits on the chain's scale, then remainders:
//                       B' to 2^-36 (an error of the state is the same in
//                       every row, so 2^-24 would show in the gradient);
//   R' = R1 + R2        R1 of 11 bits: R' to 2^-24.
// The tensor cores add FP16 products into FP32 accumulators by truncation.  A
// plain hi + lo split so loses half a unit in the last place, always toward
// zero, with every addition: z comes out 4e-8 to 1e-7 too small, and what the
// rows then add up is the log-density off by 1e-7 (FP32 arithmetic: 2e-8) and
// the gradient by 8e-7 (3e-7).  Here the leading products X1 B1 and X1 R1 are
// sums of integers below 2^24, exact in any order, in an accumulator of their
// own; what remains above 2^-24,
//   X2 B1 + X1 B2 + X3 B1 + X2 B2 + X1 B3   and   X2 R1 + X1 R2 + X3 R1 + X2 R2,
// goes to others, 2^-7 of the first, whose truncation does not matter.  Z adds
// them in FP32 once; G's are drained into FP32 registers every kDrain tiles.
//
// The slices of an X tile lie behind one another in shared memory, so that
// one MMA takes several as its N dimension: per 16 features, B1 [X1 X2 X3]
// (N = 192), B2 [X1 X2] (N = 128) and B3 X1 (N = 64) make the six products,
// into the accumulator of X1 B1 and two for the rest.  Only the first has two
// buffers (R^T is written over it for G to read); the rest is free again as
// soon as the epilogue has loaded it.  The two buffers lie on either side of
// it, so tiles alternate between the slice orders X1 X2 X3 and X3 X2 X1:
//   TMEM columns   0 Z even | 64 rest | 128 rest | 192 Z odd | 256 G | 384 G rest
//
// Warps: 0 loads X by TMA, 1 issues the MMAs of Z, 2 those of G, and 16 run the
// epilogue; two issuers, because beside the epilogue an MMA of this size costs
// its thread 80-100 clocks to issue, more than it runs.  B stays in shared
// memory.  Every wait is bounded.
//
// What bounds it: the round trip of a Z buffer (its MMAs, the epilogue, G's
// MMAs, the next load of X: the slices of B leave room for two stages above 64
// features).  Measured (log-density and gradient with the split reduction):
// 1e5 x 100, 1024 chains 849 us in FP32 arithmetic (logreg_f32.cu), 226 here.
// Errors against 64 bits there: log-density 2.2e-8 in both (the bias of the
// hardware's ex2, lg2 and rcp, which are used alike), gradient 1.2e-7 (FP32:
// 2.9e-7).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <memory>
#include <vector>

#include "engine.h"
#include "split_reduce.cuh"
#include "tc_common.cuh"
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr int kCT = 128;                    // chains per tile
constexpr int kRT = 64;                     // rows per tile
constexpr int kEpi = 16;                    // epilogue warps: 4 lane quarters x 4 row blocks
constexpr int kThreads = 32 * (3 + kEpi);
constexpr int kDrain = 4;                   // tiles between drains of G
constexpr float kNeg2Log2e = -2.8853900817779268f;  // -2 log2(e)
constexpr float kLn2 = 0.6931471805599453f;

// X', B' and R' are at most 2^15, X1 a multiple of 2^9 (6 bits), B1 and R1 of
// 2^4 (11 bits): at the top of FP16's range, so that the last slices do not
// become subnormal.
constexpr int kTop = 15;
constexpr float kRScale = 32768.f;                   // 2^kTop
constexpr float kRoundX = 12582912.f * 512.f;        // 1.5 2^23 2^9: adding it rounds to 2^9
constexpr float kRoundB = 12582912.f * 16.f;         // ... to 2^4

// TMEM columns: Z of even and odd tiles, the rest of Z, G and its rest.
constexpr uint32_t kZEven = 0, kZRest = 64, kZOdd = 192, kGA = 256, kGB = 384;

constexpr int kXBox = 8192;                 // [64 rows][128 B]: 64 features of a slice
constexpr int kStride = 129;                // floats per row of the gradient staging tile

// Shared memory for NKB blocks of 64 features.
template <int NKB>
struct Layout {
  static constexpr int kStages = NKB == 1 ? 4 : 2;      // even: tile parity = stage parity
  static constexpr int kBSlice = NKB * 16384;           // [NKB][128 chains][128 B]
  static constexpr int kXBlock = 3 * kXBox;             // the slices of 64 features
  static constexpr int kXStage = NKB * kXBlock;         // [NKB][3 slices][64 rows][128 B]
  static constexpr int kX = 3 * kBSlice;
  static constexpr int kY = kX + kStages * kXStage;     // y - 1/2 scaled, [stages][64]
  static constexpr int kExp = kY + kStages * kRT * 4;   // exponent of each chain's states
  static constexpr int kCtl = kExp + kCT * 4;
  static constexpr int kBytes = kCtl + 256 + 1024;
  // After the last load the X stages hold the gradient tile and the row
  // blocks' log-likelihoods.
  static_assert(kCT * kStride * 4 + 4 * kCT * 8 <= kStages * kXStage, "staging fits the X stages");
  static_assert(kBytes <= 232448, "shared memory over the sm_103a limit");
};

struct Bars {
  uint64_t x_full[4], x_empty[4], z_full[2], r_full[2], zr_free[2], rest_free, g_full, g_free;
  uint64_t drain[2];
};

// floor(log2 |v|); -127 for zero and subnormals, 128 for infinities and NaN.
__host__ __device__ inline int float_exponent(uint32_t bits) {
  return (int)((bits >> 23) & 255u) - 127;
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// -copysign(w, h): the magnitude of w with the sign of -h.
__device__ __forceinline__ float neg_copysign(float w, float h) {
  return __int_as_float((__float_as_int(w) & 0x7fffffff) |
                        (~__float_as_int(h) & (int)0x80000000));
}

// Two Kahan sums at once.
struct Kahan2 {
  float2 sum, comp;
  __device__ __forceinline__ void add(float2 x) {
    const float2 minus = f2(-1.f, -1.f);
    const float2 v = __ffma2_rn(comp, minus, x);
    const float2 t = __fadd2_rn(sum, v);
    comp = __ffma2_rn(v, minus, __ffma2_rn(sum, minus, t));
    sum = t;
  }
  __device__ __forceinline__ double total() const {
    return ((double)sum.x - (double)comp.x) + ((double)sum.y - (double)comp.y);
  }
};

// 16 rows of one chain, two at a time.  h is z / 2 over the power of two in ks
// = -2 log2(e) 2^k.  With arg = ks |h|, t = 2^arg = e^-|z| and u = 1 + t:
//   acc += |z| / 2 + ln u, where |z| / 2 = -arg / (2 log2 e) and one lg2 takes the
//   product of four rows' u (the FP32 kernel's sums, to rounding);
//   R' = 2^15 ((y - 1/2) - sign(z) (1/u - 1/2)) (rcp.approx, within one ulp),
// in slices, packed: R1 in r[0..7], R2 in r[8..15].
// MASK: rows at or past `nvalid` are padding (X = 0) and leave acc unchanged.
template <bool MASK>
__device__ __forceinline__ void rows16(const float (&h)[16], const float* __restrict__ ys,
                                       int nvalid, float ks, Kahan2* acc, uint32_t (&r)[16]) {
  const float2 one = f2(1.f, 1.f), scale = f2(kRScale, kRScale);
  const float2 mhalf = f2(-0.5f * kRScale, -0.5f * kRScale);
  const float2 up = f2(kRoundB, kRoundB), down = f2(-kRoundB, -kRoundB), minus = f2(-1.f, -1.f);
  // -1 / (2 log2 e), the reciprocal of the constant in ks, in two floats (one
  // would be off by 1e-8, the same way in every row).
  constexpr double kInv = 1.0 / (double)kNeg2Log2e;
  constexpr float kHi = (float)kInv, kLo = (float)(kInv - (double)kHi);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float s4[2], l4[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int g = 2 * half + q;
      float2 sa = f2(0.f, 0.f), pr = one;
      const float4 yv = *reinterpret_cast<const float4*>(ys + 4 * g);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 4 * g + 2 * e;
        float2 arg = f2(fabsf(h[j]) * ks, fabsf(h[j + 1]) * ks);
        float2 u = __fadd2_rn(f2(tc::ex2_approx(arg.x), tc::ex2_approx(arg.y)), one);
        if (MASK) {
          if (j >= nvalid) { arg.x = 0.f; u.x = 1.f; }
          if (j + 1 >= nvalid) { arg.y = 0.f; u.y = 1.f; }
        }
        sa = e == 0 ? arg : __fadd2_rn(sa, arg);
        pr = e == 0 ? u : __fmul2_rn(pr, u);
        const float2 w = __ffma2_rn(f2(tc::rcp_approx(u.x), tc::rcp_approx(u.y)), scale, mhalf);
        const float2 ym = e == 0 ? f2(yv.x, yv.y) : f2(yv.z, yv.w);
        const float2 rv = __fadd2_rn(ym, f2(neg_copysign(w.x, h[j]), neg_copysign(w.y, h[j + 1])));
        const float2 r1 = __fadd2_rn(__fadd2_rn(rv, up), down);
        const float2 r2 = __ffma2_rn(r1, minus, rv);
        r[2 * g + e] = pack_half2(r1.x, r1.y);
        r[8 + 2 * g + e] = pack_half2(r2.x, r2.y);
      }
      s4[q] = sa.x + sa.y;
      l4[q] = tc::lg2_approx(pr.x * pr.y);
    }
    const float2 s = f2(s4[0], s4[1]);
    const float2 az = __ffma2_rn(s, f2(kHi, kHi), __fmul2_rn(s, f2(kLo, kLo)));
    acc->add(__ffma2_rn(f2(l4[0], l4[1]), f2(kLn2, kLn2), az));
  }
}

// fexp: per feature, floor(log2 max |X|); X' = X 2^(kTop - 1 - fexp).
// gscale: 2^(fexp + 1 - 2 kTop), from G' to G.
// KS: 16-feature K-steps (the MMA loops are unrolled: fewest instructions each).
template <int KS>
__global__ void __launch_bounds__(kThreads, 1)
logreg_f16_kernel(const __grid_constant__ CUtensorMap xmap1, const __grid_constant__ CUtensorMap xmap2,
                  const __grid_constant__ CUtensorMap xmap3, const float* __restrict__ ym,
                  const int* __restrict__ fexp, const float* __restrict__ gscale, int N, int D,
                  const float* __restrict__ Q, int ldq, const int* __restrict__ n_dev, int c_base,
                  int c_lim, int grid, double* __restrict__ lpart, float* __restrict__ gpart,
                  int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int n = chunk_count(*n_dev, c_base, c_lim);
  const int row_tiles = (N + kRT - 1) / kRT;
  const int S = split_count(n, kCT, kRT, grid, N);
  const int tiles = (n + kCT - 1) / kCT;
  if (S == 0 || (int)blockIdx.x >= tiles * S) return;
  const int tile = blockIdx.x % tiles, split = blockIdx.x / tiles;
  const int c0 = tile * kCT;
  const int rt_begin = (int)((long long)split * row_tiles / S);
  const int rt_end = (int)((long long)(split + 1) * row_tiles / S);
  const int T = rt_end - rt_begin;
  constexpr int nkb = (KS + 3) / 4;            // 64-feature blocks
  using L = Layout<nkb>;
  constexpr int kStages = L::kStages;

  unsigned char* Bs = smem;
  unsigned char* Xs = smem + L::kX;
  float* Ys = reinterpret_cast<float*>(smem + L::kY);
  int* cexp = reinterpret_cast<int*>(smem + L::kExp);
  Bars* bars = reinterpret_cast<Bars*>(smem + L::kCtl);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kCtl + sizeof(Bars));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      tc::mbar_init(&bars->x_full[i], 1);
      tc::mbar_init(&bars->x_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars->z_full[i], 1);
      tc::mbar_init(&bars->r_full[i], kEpi);
      tc::mbar_init(&bars->zr_free[i], 1);
    }
    tc::mbar_init(&bars->rest_free, kEpi);
    tc::mbar_init(&bars->g_full, 1);
    tc::mbar_init(&bars->g_free, kEpi);
    for (int i = 0; i < 2; ++i) tc::mbar_init(&bars->drain[i], 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
    tc::prefetch_tmap(&xmap1);
    tc::prefetch_tmap(&xmap2);
    tc::prefetch_tmap(&xmap3);
  }
  if (warp == 1) tc::tmem_alloc(tmem_slot, 512);
  // Chain states -> B1, B2, B3, K-major 128-byte-swizzled [NKB][128][128 B]: a warp
  // per chain, four features per lane.  B' = q 2^(fexp + kTop - 1 - mexp) is
  // below 2^kTop, with mexp the largest exponent of the chain's states in
  // the scaled features.  Its limits keep the powers of two used with it
  // normal floats (z beyond them is outside float's range, or 2^-80 of nothing).
  {
    const int d0 = 4 * lane;
    int fe[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) fe[j] = d0 + j < D ? fexp[d0 + j] : 0;
    for (int cc = warp; cc < kCT; cc += kThreads / 32) {
      float v[4];
      int ex = -1024;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = (c0 + cc < n && d0 + j < D) ? Q[(size_t)(c0 + cc) * ldq + d0 + j] : 0.f;
        if (v[j] != 0.f) ex = max(ex, float_exponent(__float_as_uint(v[j])) + fe[j]);
      }
      const int mexp = max(-96, min(140, __reduce_max_sync(0xffffffffu, ex)));
      float b1[4], b2[4], b3[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float b = v[j] != 0.f ? ldexpf(v[j], fe[j] + kTop - 1 - mexp) : 0.f;
        b1[j] = __fadd_rn(__fadd_rn(b, kRoundB), -kRoundB);
        b2[j] = b - b1[j];
        b3[j] = b2[j] - __half2float(__float2half_rn(b2[j]));
      }
      if (lane == 0) cexp[cc] = mexp;
      if (d0 >= nkb * 64) continue;
      const uint32_t off = (d0 >> 6) * 16384 + tc::sw128_offset(cc, d0 & 63);
      *reinterpret_cast<uint2*>(Bs + off) =
          make_uint2(pack_half2(b1[0], b1[1]), pack_half2(b1[2], b1[3]));
      *reinterpret_cast<uint2*>(Bs + L::kBSlice + off) =
          make_uint2(pack_half2(b2[0], b2[1]), pack_half2(b2[2], b2[3]));
      *reinterpret_cast<uint2*>(Bs + 2 * L::kBSlice + off) =
          make_uint2(pack_half2(b3[0], b3[1]), pack_half2(b3[2], b3[3]));
    }
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Shared-memory descriptors are linear in the start address (bits 0-13 hold
  // address >> 4, and every operand lies below 256 KB): base descriptors plus
  // compile-time offsets.
  const uint64_t bk = tc::smem_desc_sw128(tc::smem_u32(Bs), 16, 1024);     // B, K-major
  const uint64_t xk = tc::smem_desc_sw128(tc::smem_u32(Xs), 16, 1024);     // X, K-major
  const uint64_t xmn = tc::smem_desc_sw128(tc::smem_u32(Xs), L::kXBlock, 1024);  // MN-major
  constexpr uint64_t kB2 = L::kBSlice >> 4, kB3 = 2 * L::kBSlice >> 4, kBox = kXBox >> 4;
  if (warp == 0) {
    // ---------------- TMA loads of X ----------------
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)L::kXStage + kRT * 4u;
      int it = 0;
      for (; it < T; ++it) {
        const int s = it % kStages;
        if (!wait_or_abort(&bars->x_empty[s], ((uint32_t)(it / kStages) & 1) ^ 1, abort_flag)) {
          tc::record_error(err, kTcTimeoutTma);
          *abort_flag = 1;
          break;
        }
        const int r0 = (rt_begin + it) * kRT;
        tc::mbar_arrive_expect_tx(&bars->x_full[s], bytes);
        unsigned char* xs = Xs + s * L::kXStage;
        const int first = it & 1 ? 2 * kXBox : 0, last = it & 1 ? 0 : 2 * kXBox;   // X1, X3
#pragma unroll
        for (int kb = 0; kb < nkb; ++kb) {
          unsigned char* xb = xs + kb * L::kXBlock;
          tc::tma_load_2d(xb + first, &xmap1, kb * 64, r0, &bars->x_full[s]);
          tc::tma_load_2d(xb + kXBox, &xmap2, kb * 64, r0, &bars->x_full[s]);
          tc::tma_load_2d(xb + last, &xmap3, kb * 64, r0, &bars->x_full[s]);
        }
        tc::bulk_load(Ys + s * kRT, ym + r0, kRT * 4u, &bars->x_full[s]);
      }
      // Every issued load has landed before the CTA can exit.
      for (int j = (it > kStages ? it - kStages : 0); j < it; ++j)
        tc::mbar_wait(&bars->x_full[j % kStages], (uint32_t)((j / kStages) & 1), kWaitLimitNs);
    }
  } else if (warp == 1) {
    // ---------------- the MMAs of Z ----------------
    if (lane == 0) {
      constexpr uint32_t idesc3 = tc::idesc_16bit_f32(128, 3 * kRT, false, false, false);
      constexpr uint32_t idesc2 = tc::idesc_16bit_f32(128, 2 * kRT, false, false, false);
      constexpr uint32_t idesc1 = tc::idesc_16bit_f32(128, kRT, false, false, false);
      bool ok = true;
      for (int it = 0; it < T; ++it) {
        const int s = it % kStages, odd = it & 1;
        // R of tile it - 2 has been read, the rest of tile it - 1 loaded.
        if ((it >= 2 && !wait_or_abort(&bars->zr_free[odd], ((uint32_t)(it >> 1) & 1) ^ 1,
                                       abort_flag)) ||
            (it >= 1 && !wait_or_abort(&bars->rest_free, ((uint32_t)it & 1) ^ 1, abort_flag)) ||
            !wait_or_abort(&bars->x_full[s], (uint32_t)(it / kStages) & 1, abort_flag)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint64_t x3 = xk + (uint64_t)((s * L::kXStage) >> 4);   // all three slices
        const uint64_t x12 = x3 + (odd ? kBox : 0);                   // X1 and X2, either order
        const uint64_t x1 = x3 + (odd ? 2 * kBox : 0);
        const uint32_t tz = tmem + (odd ? kZRest : kZEven);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          const uint64_t bd = bk + (uint64_t)(((k >> 2) * 16384 + (k & 3) * 32) >> 4);
          const uint64_t xo = (uint64_t)(((k >> 2) * L::kXBlock + (k & 3) * 32) >> 4);
          tc::mma_16bit(tz, bd, x3 + xo, idesc3, k > 0 ? 1u : 0u);
          tc::mma_16bit(tmem + kZRest, bd + kB2, x12 + xo, idesc2, 1u);
          tc::mma_16bit(tmem + kZRest, bd + kB3, x1 + xo, idesc1, 1u);
        }
        tc::mma_commit(&bars->z_full[odd]);
      }
      if (!ok) {
        tc::record_error(err, kTcTimeoutMma);
        *abort_flag = 1;
      }
      // This thread's MMAs have completed before the CTA exits.
      tc::mma_commit(&bars->drain[0]);
      tc::mbar_wait(&bars->drain[0], 0, kWaitLimitNs);
    }
  } else if (warp == 2) {
    // ---------------- the MMAs of G ----------------
    if (lane == 0) {
      constexpr uint32_t idesc_g = tc::idesc_16bit_f32(128, KS * 16, false, true, false);
      bool ok = true;
      int drained = 0;       // drains of G the epilogue has to have done
      for (int it = 0; it < T; ++it) {
        const int s = it % kStages, odd = it & 1;
        const bool fresh = it % kDrain == 0;
        if (!wait_or_abort(&bars->r_full[odd], (uint32_t)(it >> 1) & 1, abort_flag) ||
            (fresh && it > 0 &&
             !wait_or_abort(&bars->g_free, (uint32_t)drained++ & 1, abort_flag))) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint64_t xs = xmn + (uint64_t)((s * L::kXStage) >> 4);
        const uint64_t x1 = xs + (odd ? 2 * kBox : 0), x2 = xs + kBox, x3 = xs + (odd ? 0 : 2 * kBox);
        // 16 rows of R take 16 columns: 8 of R1, 8 of R2.
        const uint32_t tr = tmem + (odd ? kZOdd : kZEven);
#pragma unroll
        for (int ks = 0; ks < kRT / 16; ++ks) {
          const uint32_t ra = tr + ks * 16;
          const uint64_t xo = (uint64_t)((ks * 2048) >> 4);
          const uint32_t acc = fresh && ks == 0 ? 0u : 1u;
          tc::mma_16bit_tmem_a(tmem + kGA, ra, x1 + xo, idesc_g, acc);
          tc::mma_16bit_tmem_a(tmem + kGB, ra, x2 + xo, idesc_g, acc);
          tc::mma_16bit_tmem_a(tmem + kGB, ra + 8, x1 + xo, idesc_g, 1u);
          tc::mma_16bit_tmem_a(tmem + kGB, ra, x3 + xo, idesc_g, 1u);
          tc::mma_16bit_tmem_a(tmem + kGB, ra + 8, x2 + xo, idesc_g, 1u);
        }
        tc::mma_commit(&bars->zr_free[odd]);
        tc::mma_commit(&bars->x_empty[s]);
        if (it + 1 == T || (it + 1) % kDrain == 0) tc::mma_commit(&bars->g_full);
      }
      if (!ok) {
        tc::record_error(err, kTcTimeoutMma);
        *abort_flag = 1;
      }
      tc::mma_commit(&bars->drain[1]);
      tc::mbar_wait(&bars->drain[1], 0, kWaitLimitNs);
    }
  } else {
    // ---------------- epilogue (16 warps) ----------------
    const int quarter = warp & 3;                // TMEM lanes 32*quarter .. (chains)
    const int rblk = (warp - 3) >> 2;            // rows [16 rblk, +16), features [32 rblk, +32)
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int c = quarter * 32 + lane;           // chain of this thread
    // X B^T / 2 = X' B'^T 2^(mexp + 1 - 2 kTop)
    const float ks = kNeg2Log2e * __int_as_float((cexp[c] + 1 - 2 * kTop + 127) << 23);
    // Kahan sum over tiles of sum_r (|z_r| / 2 + ln(1 + e^-|z_r|)) for this
    // chain's rows; the linear part sum_r (y_r - 1/2) z_r is added exactly by
    // the reduction.
    Kahan2 acc{f2(0.f, 0.f), f2(0.f, 0.f)};
    float g[32];             // G drained so far (this chain's 32 features)
    int drained = 0;
    bool ok = true;
    auto drain = [&]() {     // G of the tiles since the last drain
      if (!warp_wait(&bars->g_full, (uint32_t)drained & 1, abort_flag)) return false;
      tc::tc_fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float va[16], vb[16];
        const uint32_t col = tmem + lane_base + rblk * 32 + half * 16;
        tc::tmem_ld16(col + kGA, va);
        tc::tmem_ld16(col + kGB, vb);
        tc::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float v = va[j] + vb[j];
          g[half * 16 + j] = drained == 0 ? v : g[half * 16 + j] + v;
        }
      }
      ++drained;
      return true;
    };
    for (int it = 0; it < T; ++it) {
      const int s = it % kStages, odd = it & 1;
      if (!warp_wait(&bars->z_full[odd], (uint32_t)(it >> 1) & 1, abort_flag)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      const uint32_t col = tmem + lane_base + rblk * 16, tz = col + (odd ? kZOdd : kZEven);
      float h[16], ha[16], hb[16];
      tc::tmem_ld16(tz, h);
      tc::tmem_ld16(col + kZRest, ha);
      tc::tmem_ld16(col + kZRest + kRT, hb);
      tc::tmem_ld_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars->rest_free);
#pragma unroll
      for (int j = 0; j < 16; ++j) h[j] += ha[j] + hb[j];
      // y of this tile: landed with X (already complete; the wait makes the
      // bulk copy's writes visible to this thread).
      if (!warp_wait(&bars->x_full[s], (uint32_t)(it / kStages) & 1, abort_flag)) {
        ok = false;
        break;
      }
      const int nvalid = N - ((rt_begin + it) * kRT + rblk * 16);
      const float* ys = Ys + s * kRT + rblk * 16;
      uint32_t r[16];
      if (nvalid >= 16) rows16<false>(h, ys, 16, ks, &acc, r);
      else rows16<true>(h, ys, nvalid, ks, &acc, r);
      tc::tmem_st16(tz, r);
      tc::tmem_st_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars->r_full[odd]);
      // The previous group's G, one tile late: its MMAs run beside this tile.
      if (it > 0 && it % kDrain == 0) {
        if (!drain()) {
          ok = false;
          break;
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bars->g_free);
      }
    }
    if (ok && T > 0) ok = drain();
    float* stage = reinterpret_cast<float*>(Xs);                      // [128][kStride]
    double* red = reinterpret_cast<double*>(Xs + kCT * kStride * 4);  // [4][128]
    if (!ok) {
      tc::record_error(err, kTcTimeoutEpilogue);
      *abort_flag = 1;
    } else {
      // The X stages are idle: every load has been consumed by finished MMAs.
      float* dst = stage + c * kStride + rblk * 32;
#pragma unroll
      for (int j = 0; j < 32; ++j) dst[j] = g[j];
      red[rblk * kCT + c] = -acc.total();
    }
    named_barrier(1, 32 * kEpi);
    if (ok) {
      const int et = tid - 96;
      if (et < kCT && c0 + et < n)
        lpart[(size_t)split * n + c0 + et] =
            red[et] + red[kCT + et] + red[2 * kCT + et] + red[3 * kCT + et];
      // Coalesced gradient partials: one warp per chain row at a time.
      for (int cc = warp - 3; cc < kCT; cc += kEpi) {
        if (c0 + cc >= n) break;
        float* row = gpart + ((size_t)split * n + c0 + cc) * D;
        for (int d = lane; d < D; d += 32) row[d] = stage[cc * kStride + d] * gscale[d];
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 512);
  }
}

// ---- data preparation ----
// Largest |x| of each column, as bits.
__global__ void column_max_kernel(const float* __restrict__ X, int64_t N, int D, int64_t chunk,
                                  unsigned* __restrict__ out) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk, r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    unsigned m = 0;
#pragma unroll 8
    for (int64_t r = r0; r < r1; ++r) m = max(m, __float_as_uint(X[r * D + d]) & 0x7fffffffu);
    if (m) atomicMax(&out[d], m);
  }
}

struct Slices {
  float x1, x2, x3, rest;   // X' = x1 + x2 + x3 + rest
};

__device__ __forceinline__ Slices slice_x(float x, int fexp) {
  const float v = ldexpf(x, kTop - 1 - fexp);
  Slices s;
  s.x1 = __fadd_rn(__fadd_rn(v, kRoundX), -kRoundX);
  s.x2 = __half2float(__float2half_rn(v - s.x1));
  const float r2 = (v - s.x1) - s.x2;
  s.x3 = __half2float(__float2half_rn(r2));
  s.rest = r2 - s.x3;
  return s;
}

// Sums of X'^2 and of what the slices leave of it, squared, over rows
// [b chunk, (b + 1) chunk) into part[b][d], in a fixed order.
__global__ void column_rest_kernel(const float* __restrict__ X, int64_t N, int D, int64_t chunk,
                                   const unsigned* __restrict__ max_bits,
                                   float2* __restrict__ part) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk, r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const int fe = float_exponent(max_bits[d]);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int64_t r = r0; r < r1; ++r) {
      const Slices s = slice_x(X[r * D + d], fe);
      const float v = s.x1 + s.x2 + s.x3;
      acc.x = fmaf(v, v, acc.x);
      acc.y = fmaf(s.rest, s.rest, acc.y);
    }
    part[(size_t)blockIdx.x * D + d] = acc;
  }
}

// One block per feature, fixed order.
__global__ void __launch_bounds__(128)
column_rest_sum(const float2* __restrict__ part, int nb, int D, double2* __restrict__ out) {
  __shared__ double2 sh[128];
  const int d = blockIdx.x, tid = threadIdx.x;
  double2 acc = make_double2(0.0, 0.0);
  for (int b = tid; b < nb; b += 128) {
    acc.x += (double)part[(size_t)b * D + d].x;
    acc.y += (double)part[(size_t)b * D + d].y;
  }
  sh[tid] = acc;
  for (int o = 64; o > 0; o >>= 1) {
    __syncthreads();
    if (tid < o) {
      sh[tid].x += sh[tid + o].x;
      sh[tid].y += sh[tid + o].y;
    }
  }
  if (tid == 0) out[d] = sh[0];
}

// X [N][D] -> X1, X2, X3 [N][Dp], zero-padded features.
__global__ void f16_split_kernel(const float* __restrict__ X, int64_t N, int D, int Dp,
                                 const int* __restrict__ fexp, __half* __restrict__ x1,
                                 __half* __restrict__ x2, __half* __restrict__ x3) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * Dp) return;
  const int64_t r = i / Dp;
  const int d = (int)(i - r * Dp);
  Slices s{0.f, 0.f, 0.f, 0.f};
  if (d < D) s = slice_x(X[r * D + d], fexp[d]);
  x1[i] = __float2half_rn(s.x1);
  x2[i] = __float2half_rn(s.x2);
  x3[i] = __float2half_rn(s.x3);
}

// ym = (y - 1/2) 2^15, zero past N.
__global__ void f16_labels_kernel(const float* __restrict__ y, int64_t N, int64_t padded,
                                  float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < padded) out[i] = i < N ? (y[i] - 0.5f) * kRScale : 0.f;
}

// lin[d] = sum_r (y_r - 1/2) X[r][d] in float64 and a fixed order: block b
// sums rows [b chunk, (b + 1) chunk) into part[b][d]; blocks added in order.
__global__ void f16_lin_partial(const float* __restrict__ X, const float* __restrict__ y,
                                int64_t N, int D, int64_t chunk, double* __restrict__ part) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk;
  const int64_t r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    double acc = 0.0;
    for (int64_t r = r0; r < r1; ++r) acc += ((double)y[r] - 0.5) * (double)X[r * D + d];
    part[(size_t)blockIdx.x * D + d] = acc;
  }
}

__global__ void f16_lin_sum(const double* __restrict__ part, int nb, int D,
                            double* __restrict__ lin) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  double acc = 0.0;
#pragma unroll 16
  for (int b = 0; b < nb; ++b) acc += part[(size_t)b * D + d];
  lin[d] = acc;
}

typedef decltype(&logreg_f16_kernel<1>) Kernel;

// Fewer rows stay with the FP32 kernel.  A log-density of either kernel is a
// float64 sum of float32 terms whose rounding averages out over the rows: the
// two kernels' differ by 6e-10 of it at 1e5 rows, 7e-10 at 65,536 and 1.1e-9 at
// 32,768 (100 features).  Runs are resumed from stored log-densities and
// compared with earlier ones, to 1e-9.
constexpr int64_t kF16MinRows = 65536;

class LogregF16 final : public Target {
 public:
  LogregF16(gbm_context* ctx, const float* X, int64_t n, int64_t d, const float* y,
            float prior_scale, const std::vector<int>& fexp)
      : N_(n), D_(d) {
    dim = d;
    const int Dp = (int)((d + 15) / 16 * 16);   // a box's features past it read as zeros
    const int64_t padded = (n + kRT - 1) / kRT * kRT;
    cudaStream_t s = ctx->stream;
    for (auto& b : x_) b.reserve(sizeof(__half) * (size_t)N_ * Dp);
    ym_.reserve(sizeof(float) * (size_t)padded);
    std::vector<float> gs(d);
    for (int64_t i = 0; i < d; ++i) gs[i] = std::ldexp(1.f, fexp[i] + 1 - 2 * kTop);
    fexp_.reserve(sizeof(int) * d);
    gscale_.reserve(sizeof(float) * d);
    GBM_CUDA(cudaMemcpyAsync(fexp_.ptr, fexp.data(), sizeof(int) * d, cudaMemcpyHostToDevice, s));
    GBM_CUDA(cudaMemcpyAsync(gscale_.ptr, gs.data(), sizeof(float) * d, cudaMemcpyHostToDevice,
                             s));
    const int64_t total = N_ * Dp;
    f16_split_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
        X, N_, (int)D_, Dp, fexp_.as<int>(), x_[0].as<__half>(), x_[1].as<__half>(),
        x_[2].as<__half>());
    f16_labels_kernel<<<(unsigned)((padded + 255) / 256), 256, 0, s>>>(y, N_, padded,
                                                                       ym_.as<float>());
    GBM_CUDA(cudaGetLastError());
    {
      const int nb = 2 * ctx->num_sms;
      const int64_t chunk = (N_ + nb - 1) / nb;
      DeviceBuffer part;
      part.reserve(sizeof(double) * (size_t)nb * D_);
      lin_.reserve(sizeof(double) * (size_t)D_);
      f16_lin_partial<<<nb, 128, 0, s>>>(X, y, N_, (int)D_, chunk, part.as<double>());
      f16_lin_sum<<<1, 128, 0, s>>>(part.as<double>(), nb, (int)D_, lin_.as<double>());
      GBM_CUDA(cudaGetLastError());
      GBM_CUDA(cudaStreamSynchronize(s));   // `part`, `gs` end here
    }
    inv_var_ = 1.f / (prior_scale * prior_scale);
    log_norm_ = -log((double)prior_scale) - 0.5 * log(2.0 * M_PI);
    grid_ = ctx->num_sms;
    err_dev_ = ctx->err_dev;
    for (int i = 0; i < 3; ++i) encode_rows(&xmap_[i], x_[i].ptr, N_, Dp, kRT);
    const Kernel fns[8] = {logreg_f16_kernel<1>, logreg_f16_kernel<2>, logreg_f16_kernel<3>,
                           logreg_f16_kernel<4>, logreg_f16_kernel<5>, logreg_f16_kernel<6>,
                           logreg_f16_kernel<7>, logreg_f16_kernel<8>};
    kernel_ = fns[(d - 1) / 16];
    smem_ = Dp <= 64 ? Layout<1>::kBytes : Layout<2>::kBytes;
    GBM_CUDA(cudaFuncSetAttribute(kernel_, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_));
  }

  size_t workspace_bytes(int64_t cap) const override {
    const size_t rows = (size_t)grid_ * kCT + (size_t)cap;
    return rows * sizeof(double) + rows * (size_t)D_ * sizeof(float) + 256;
  }

  // One launch covers at most grid_ * 128 chains (one work item per CTA);
  // larger batches run as consecutive chunks that share the workspace.
  void eval(const float* q, int ldq, const int* n_dev, int cap, double* logp, float* grad,
            int ldg, void* ws, cudaStream_t s) override {
    const size_t rows = (size_t)grid_ * kCT + (size_t)cap;
    double* lpart = static_cast<double*>(ws);
    float* gpart = reinterpret_cast<float*>(lpart + rows);
    const int N = (int)N_, D = (int)D_;
    const int lim = grid_ * kCT;
    for (int base = 0; base < cap; base += lim) {
      const float* qc = q + (size_t)base * ldq;
      const int g = work_grid(grid_, std::min(lim, cap - base), kCT, N_, kMinSplitRows);
      kernel_<<<g, kThreads, smem_, s>>>(
          xmap_[0], xmap_[1], xmap_[2], ym_.as<float>(), fexp_.as<int>(), gscale_.as<float>(), N,
          D, qc, ldq, n_dev, base, lim, g, lpart, gpart, err_dev_);
      GBM_CUDA(cudaGetLastError());
      launch_split_reduce(lpart, gpart, qc, ldq, n_dev, base, lim, std::min(lim, cap - base), kCT,
                          kRT, g, N, D, inv_var_, log_norm_, lin_.as<double>(), logp + base,
                          grad + (size_t)base * ldg, ldg, s);
    }
  }

  int launches_per_eval(int64_t cap) const override {
    return 2 * (int)((cap + (int64_t)grid_ * kCT - 1) / ((int64_t)grid_ * kCT));
  }
  double flops(int64_t n) const override { return 4.0 * (double)N_ * D_ * n; }
  double bytes(int64_t n) const override {
    return 4.0 * (double)N_ * D_ + 4.0 * N_ + 8.0 * (double)n * D_ + 8.0 * n;
  }

 private:
  int64_t N_, D_;
  int grid_ = 0, smem_ = 0;
  float inv_var_ = 1.f;
  double log_norm_ = 0.0;
  int* err_dev_ = nullptr;
  DeviceBuffer x_[3], ym_, fexp_, gscale_, lin_;
  CUtensorMap xmap_[3];
  Kernel kernel_ = nullptr;
};

}  // namespace

std::unique_ptr<Target> make_logreg_f16(gbm_context* ctx, const float* X, int64_t n, int64_t d,
                                        const float* y, float prior_scale) {
  if (d > 128 || n < kF16MinRows) return nullptr;
  const int nb = 8 * ctx->num_sms;
  const int64_t chunk = (n + nb - 1) / nb;
  const size_t off_part = 1024;
  const size_t off_sum = off_part + (sizeof(float2) * (size_t)nb * d + 255) / 256 * 256;
  DeviceBuffer buf;
  buf.reserve(off_sum + sizeof(double2) * d);
  unsigned* mx = buf.as<unsigned>();
  float2* part = reinterpret_cast<float2*>(buf.as<char>() + off_part);
  double2* sum = reinterpret_cast<double2*>(buf.as<char>() + off_sum);
  cudaStream_t s = ctx->stream;
  GBM_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned) * d, s));
  column_max_kernel<<<nb, 128, 0, s>>>(X, n, (int)d, chunk, mx);
  column_rest_kernel<<<nb, 128, 0, s>>>(X, n, (int)d, chunk, mx, part);
  column_rest_sum<<<(unsigned)d, 128, 0, s>>>(part, nb, (int)d, sum);
  GBM_CUDA(cudaGetLastError());
  std::vector<unsigned> hmax(d);
  std::vector<double2> hsum(d);
  GBM_CUDA(cudaMemcpyAsync(hmax.data(), mx, sizeof(unsigned) * d, cudaMemcpyDeviceToHost, s));
  GBM_CUDA(cudaMemcpyAsync(hsum.data(), sum, sizeof(double2) * d, cudaMemcpyDeviceToHost, s));
  GBM_CUDA(cudaStreamSynchronize(s));
  // The splits hold a column if what they leave of it is below 2^-26 of it, in
  // root mean square (a normal sample: 2^-30); infinities, NaN and powers of
  // two that the scaling cannot carry go to the FP32 kernel.
  // A column of zeros must not set the scale of the states.
  std::vector<int> fexp(d, -64);
  for (int64_t i = 0; i < d; ++i) {
    if (hmax[i] == 0) continue;
    fexp[i] = float_exponent(hmax[i]);
    if (fexp[i] < -60 || fexp[i] > 60 || !(hsum[i].y <= ldexp(hsum[i].x, -52))) return nullptr;
  }
  return std::unique_ptr<Target>(new LogregF16(ctx, X, n, d, y, prior_scale, fexp));
}

}  // namespace gbm
