// Gradient partials of a logistic regression on the tensor cores, from residuals
// in memory: G^T[c][d] = sum_r R[r][c] X[r][d] with R and X as FP16 hi + lo
// (f16_rows.cuh), for the FP32 targets whose features are too many for a kernel
// that also forms Z.  R is held as multiples of 2^-15, or of a power of two for each
// 32 rows of a chain, which then goes into the sums.
//
// A CTA owns 128 chains x 256 features (M x N of its MMAs) and a stretch of rows,
// and writes one partial.  TMA brings 64 rows of R and X into one of two stages;
// 6 MMAs for each 32 rows form R_lo^T X_hi + R_hi^T X_lo + R_hi^T X_hi in one of
// two accumulators (the small terms first, and few rows: the tensor cores truncate
// every addition), and eight warps add it to FP32 sums in their registers beside
// the next rows' MMAs.  Gradient error against 64 bits 6e-8 to 1.8e-7 over 300 to
// 60,000 rows, 129 to 1000 features (FP32 on the CUDA cores: 1e-7 to 2.4e-7).
//
// What bounds it: MMA issue (1,536 clocks a stage at 256 features) and as many
// bytes of R and X from L2 (96 KB a stage).  30,011 x 237, 192 chains: 27 us, half
// of it a CTA's start, first loads and partial (six stages each).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "f16_rows.cuh"
#include "split_reduce.cuh"
#include "tc_common.cuh"

namespace gbm {
namespace {

constexpr int kGradCT = 128;                // chains of a CTA
constexpr int kGradRT = 64;                 // rows of a stage
constexpr int kGradFT = 256;                // features of a CTA
constexpr int kGradDrain = 256;             // threads that add
constexpr int kGradThreads = kGradDrain + 64;
constexpr int kGradTimeoutCode = 6;
constexpr int kGradR = kGradCT * kGradRT * 2;        // hi or lo of R
constexpr int kGradXBox = 64 * kGradRT * 2;          // 64 features x 64 rows
constexpr int kGradStage = 2 * kGradR + 2 * (kGradFT / 64) * kGradXBox;
constexpr int kGradSmem = 2 * kGradStage + 256 + 1024;
static_assert(kGradSmem <= 232448, "shared memory over the sm_103a limit");
static_assert(kGradCT * (kGradFT + 1) * 4 <= 2 * kGradStage, "gradient tile fits the stages");

struct GradBars {
  uint64_t full[2], empty[2], acc_full[2], acc_empty[2];
};

// R: boxes of 64 chains x 64 rows of [N][chains] (K_MAJOR false), or of 64 rows x
// 128 chains of [chains][rows].  grid = split stretches x chain tiles at most,
// times feature tiles.  rscale (K_MAJOR false): what 2^15 R of a chain's 32 rows is
// of what is stored, [rows / 32][cp].
template <bool K_MAJOR>
__global__ void __launch_bounds__(kGradThreads, 1)
grad_tc_kernel(const __grid_constant__ CUtensorMap rhi, const __grid_constant__ CUtensorMap rlo,
               const __grid_constant__ CUtensorMap xhi, const __grid_constant__ CUtensorMap xlo,
               const float* __restrict__ gscale, const float* __restrict__ rscale, int cp, int N,
               int D, int dp, const int* __restrict__ n_dev, int c_base, int c_lim, int grid,
               int ftiles, float* __restrict__ gpart, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int n = n_dev ? chunk_count(*n_dev, c_base, c_lim) : c_lim;
  const int S = split_count(n, kGradCT, kGradRT, grid, N);
  const int tiles = (n + kGradCT - 1) / kGradCT;
  const int ft = blockIdx.x % ftiles, item = blockIdx.x / ftiles;
  if (S == 0 || item >= tiles * S) return;
  const int c0 = item % tiles * kGradCT, split = item / tiles, f0 = ft * kGradFT;
  const int units = (N + kGradRT - 1) / kGradRT;
  const int u0 = (int)((long long)split * units / S);
  const int U = (int)((long long)(split + 1) * units / S) - u0;
  const int width = min(kGradFT, dp - f0);           // features held here, a multiple of 16
  const int boxes = (width + 63) / 64;

  GradBars* bars = reinterpret_cast<GradBars*>(smem + 2 * kGradStage);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars->full[i], 1);
      tc::mbar_init(&bars->empty[i], 1);
      tc::mbar_init(&bars->acc_full[i], 1);
      tc::mbar_init(&bars->acc_empty[i], kGradDrain / 32);
    }
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 8) tc::tmem_alloc(tmem_slot, 2 * kGradFT);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 8) {
    // ---------------- loads ----------------
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)(2 * kGradR + 2 * boxes * kGradXBox);
      int u = 0;
      for (; u < U; ++u) {
        const int s = u & 1;
        if (!wait_or_abort(&bars->empty[s], ((uint32_t)(u >> 1) & 1) ^ 1, abort_flag)) {
          tc::record_error(err, kGradTimeoutCode);
          *abort_flag = 1;
          break;
        }
        unsigned char* r = smem + s * kGradStage;
        unsigned char* x = r + 2 * kGradR;
        const int r0 = (u0 + u) * kGradRT;
        tc::mbar_arrive_expect_tx(&bars->full[s], bytes);
        if (K_MAJOR) {
          tc::tma_load_2d(r, &rhi, r0, c0, &bars->full[s]);
          tc::tma_load_2d(r + kGradR, &rlo, r0, c0, &bars->full[s]);
        } else {
          for (int b = 0; b < 2; ++b) {
            tc::tma_load_2d(r + b * (kGradR / 2), &rhi, c0 + 64 * b, r0, &bars->full[s]);
            tc::tma_load_2d(r + kGradR + b * (kGradR / 2), &rlo, c0 + 64 * b, r0,
                            &bars->full[s]);
          }
        }
        for (int b = 0; b < boxes; ++b) {
          tc::tma_load_2d(x + b * kGradXBox, &xhi, f0 + 64 * b, r0, &bars->full[s]);
          tc::tma_load_2d(x + (kGradFT / 64 + b) * kGradXBox, &xlo, f0 + 64 * b, r0,
                          &bars->full[s]);
        }
      }
      // Every issued load lands before the CTA can exit.
      for (int j = u > 2 ? u - 2 : 0; j < u; ++j)
        tc::mbar_wait(&bars->full[j & 1], (uint32_t)(j >> 1) & 1, kWaitLimitNs);
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---------------- MMAs ----------------
    if (tc::elect_one()) {
      const uint32_t idesc = tc::idesc_16bit_f32(kGradCT, width, !K_MAJOR, true, false);
      bool ok = true;
      int halves = 0;               // halves whose MMAs were issued
      for (int u = 0; u < U; ++u) {
        const int s = u & 1;
        ok = wait_or_abort(&bars->full[s], (uint32_t)(u >> 1) & 1, abort_flag);
        if (!ok) break;
        const uint32_t r = tc::smem_u32(smem + s * kGradStage), x = r + 2 * kGradR;
        // A: 64 chains' boxes beside each other, or rows of K within 128 bytes.
        const uint64_t rd = K_MAJOR ? tc::smem_desc_sw128(r, 16, 1024)
                                    : tc::smem_desc_sw128(r, kGradR / 2, 1024);
        const uint64_t xd = tc::smem_desc_sw128(x, kGradXBox, 1024);
        constexpr uint64_t kRlo = kGradR >> 4, kXlo = (kGradFT / 64) * kGradXBox >> 4;
        constexpr uint64_t kRStep = (K_MAJOR ? 32 : 2048) >> 4, kXStep = 2048 >> 4;
        for (int h = 0; h < 2; ++h) {      // halves of the stage, an accumulator each
          ok = wait_or_abort(&bars->acc_empty[h], ((uint32_t)u & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc::tc_fence_after();
          const uint32_t acc = tmem + h * kGradFT;
          const uint64_t ra = rd + 2 * h * kRStep, xa = xd + 2 * h * kXStep;
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            tc::mma_16bit(acc, ra + kRlo + ks * kRStep, xa + ks * kXStep, idesc, ks > 0 ? 1u : 0u);
            tc::mma_16bit(acc, ra + ks * kRStep, xa + kXlo + ks * kXStep, idesc, 1u);
          }
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
            tc::mma_16bit(acc, ra + ks * kRStep, xa + ks * kXStep, idesc, 1u);
          tc::mma_commit(&bars->acc_full[h]);
          ++halves;
        }
        if (!ok) break;
        tc::mma_commit(&bars->empty[s]);
      }
      if (!ok) {
        tc::record_error(err, kGradTimeoutCode);
        *abort_flag = 1;
        if (halves > 0)   // the MMAs in flight end before the CTA exits
          tc::mbar_wait(&bars->acc_full[(halves - 1) & 1], (uint32_t)((halves - 1) >> 1) & 1,
                        kWaitLimitNs);
      }
    }
    __syncwarp();
  } else {
    // ---------------- sums ----------------
    // Lane = chain (32 (warp & 3) + lane), columns [128 (warp >> 2), + 128).
    const uint32_t quarter = (uint32_t)((warp & 3) * 32) << 16;
    const int col = (warp >> 2) * 128;
    float sum[128];
#pragma unroll
    for (int i = 0; i < 128; ++i) sum[i] = 0.f;
    bool ok = true;
    const int chain = c0 + (warp & 3) * 32 + lane;
    // Of a stage's two halves, and of the next stage's, which are loaded a stage ahead.
    const bool scaled = !K_MAJOR && chain < cp;
    float scale[2] = {1.f, 1.f}, next[2] = {1.f, 1.f};
    auto load_scales = [&](int unit) {
      if (scaled && unit < U) {
        const float* sc = rscale + (size_t)(2 * (u0 + unit)) * cp + chain;
        next[0] = sc[0];
        next[1] = sc[cp];
      }
    };
    load_scales(0);
    for (int u = 0; u < 2 * U; ++u) {      // half stages
      const int s = u & 1;
      if (s == 0) {
        scale[0] = next[0];
        scale[1] = next[1];
        load_scales((u >> 1) + 1);
      }
      if (!warp_wait(&bars->acc_full[s], (uint32_t)(u >> 1) & 1, abort_flag)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (col + 16 * j >= width) break;
        float v[16];
        tc::tmem_ld16(tmem + s * kGradFT + quarter + col + 16 * j, v);
        tc::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float& at = sum[16 * j + e];
          at = K_MAJOR ? at + v[e] : fmaf(v[e], s ? scale[1] : scale[0], at);
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&bars->acc_empty[s]);
    }
    if (!ok) {
      tc::record_error(err, kGradTimeoutCode);
      *abort_flag = 1;
    }
    // Every MMA has read its stage and every load has landed: the stages become
    // the gradient tile.
    named_barrier(1, kGradDrain);
    const bool good = *abort_flag == 0;
    float* tile = reinterpret_cast<float*>(smem);
    if (good) {
      const int cc = (warp & 3) * 32 + lane;
#pragma unroll
      for (int i = 0; i < 128; ++i)
        if (col + i < width) tile[cc * (kGradFT + 1) + col + i] = sum[i];
    }
    named_barrier(1, kGradDrain);
    if (good) {
      for (int cc = warp; cc < kGradCT; cc += kGradDrain / 32) {
        if (c0 + cc >= n) break;
        float* dst = gpart + ((size_t)split * n + c0 + cc) * D + f0;
        for (int f = lane; f < min(kGradFT, D - f0); f += 32)
          dst[f] = tile[cc * (kGradFT + 1) + f] * gscale[f0 + f];
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, 2 * kGradFT);
  }
}

inline int grad_tc_ftiles(int dp) { return (dp + kGradFT - 1) / kGradFT; }
// (Chain tile, split) items of a launch for up to `cap` chains: the SMs' share
// of a feature tile, and no fewer than the chain tiles.
inline int grad_tc_grid(int num_sms, int64_t cap, int64_t N, int dp) {
  const int per = std::max(1, num_sms / grad_tc_ftiles(dp));
  const int tiles = (int)((cap + kGradCT - 1) / kGradCT);
  return std::max(work_grid(per, cap, kGradCT, N, kGradRT), tiles);
}
// Rows (of D floats) that the partials of such a launch take.
inline size_t grad_tc_rows(int num_sms, int64_t cap, int dp) {
  return (size_t)std::max<int64_t>(std::max(1, num_sms / grad_tc_ftiles(dp)),
                                   (cap + kGradCT - 1) / kGradCT) * kGradCT + (size_t)cap;
}

template <bool K_MAJOR>
void grad_tc_setup() {
  GBM_CUDA(cudaFuncSetAttribute(grad_tc_kernel<K_MAJOR>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
}

// Partials of chains [c_base, c_base + cap) whose residuals are at r (hi, then lo
// at r_lo): [N][ldr] chains with rscale, or [chains][ldr] rows.
template <bool K_MAJOR>
void launch_grad_tc(const F16Rows& x, __half* r, __half* r_lo, const float* rscale, int64_t ldr,
                    int N, int D, int dp, const int* n_dev, int c_base, int c_lim, int cap,
                    int grid, float* gpart, int* err, cudaStream_t s) {
  CUtensorMap hi, lo;
  if (K_MAJOR) {
    encode_rows(&hi, r, cap, (int)ldr, kGradCT);
    encode_rows(&lo, r_lo, cap, (int)ldr, kGradCT);
  } else {
    encode_rows(&hi, r, N, (int)ldr, kGradRT);
    encode_rows(&lo, r_lo, N, (int)ldr, kGradRT);
  }
  const int ft = grad_tc_ftiles(dp);
  grad_tc_kernel<K_MAJOR><<<(unsigned)(grid * ft), kGradThreads, kGradSmem, s>>>(
      hi, lo, x.hi, x.lo, x.gscale, rscale, (int)ldr, N, D, dp, n_dev, c_base, c_lim, grid, ft,
      gpart, err);
  GBM_CUDA(cudaGetLastError());
}

}  // namespace
}  // namespace gbm
