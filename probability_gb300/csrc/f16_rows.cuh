// X as FP16 hi + lo of scaled features, for gradient products on the tensor
// cores: X' = X 2^(kF16Top - exponent of the column's largest), and residuals
// as hi + lo of R' = kF16Scale R; gscale turns a product of the two back.  hi + lo
// carries a float to 2^-23 of itself, and not below 2^-25 (half of FP16's smallest
// step): an entry 2^16 below its column's largest loses bits, one 2^39 below is gone.
// prepare() measures what the entries lose and holds only columns that lose nothing
// to speak of.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "engine.h"
#include "tc_common.cuh"

namespace gbm {
namespace {

constexpr float kF16Scale = 32768.f;        // R' = 2^15 R
constexpr int kF16Top = 14;                 // X' < 2^15
// Rows from which targets of up to 128 and of more than 256 features hold pairs; each
// says why (between the two they are held at any number: the kernel that they
// replace is the slower and the less exact one at every size, 300 x 130 x 16 chains
// 61 against 40 us).
constexpr int64_t kPairRows = 4096;

__device__ __forceinline__ int float_exponent(unsigned bits) {
  return (int)((bits >> 23) & 255u) - 127;
}

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

// What hi + lo leaves of a column's nonzero entries, each relative to the entry:
// the largest, the sum of the others, and their number.
struct ColumnLoss {
  float rest, most;
  unsigned entries;
  __device__ __forceinline__ void add(float loss) {
    rest += fminf(loss, most);
    most = fmaxf(loss, most);
  }
};

// X [N][D] -> X' = X 2^(kF16Top - exponent of the column's largest) as FP16 hi
// + lo [N][Dp], zero-padded, and what rows [b chunk, (b + 1) chunk) lose by it in
// part[b][d].
__global__ void f16_pack_kernel(const float* __restrict__ X, int64_t N, int D, int Dp,
                                int64_t chunk, const unsigned* __restrict__ max_bits,
                                __half* __restrict__ hi, __half* __restrict__ lo,
                                ColumnLoss* __restrict__ part) {
  const int64_t r0 = (int64_t)blockIdx.x * chunk, r1 = r0 + chunk < N ? r0 + chunk : N;
  for (int d = threadIdx.x; d < Dp; d += blockDim.x) {
    const int shift = d < D ? kF16Top - float_exponent(max_bits[d]) : 0;
    ColumnLoss loss{0.f, 0.f, 0u};
#pragma unroll 4
    for (int64_t r = r0; r < r1; ++r) {
      const float x = d < D ? X[r * D + d] : 0.f;
      const float v = ldexpf(x, shift);
      const __half h = __float2half_rn(v);
      const float rest = v - __half2float(h);
      const __half l = __float2half_rn(rest);
      hi[r * Dp + d] = h;
      lo[r * Dp + d] = l;
      const float left = fabsf(rest - __half2float(l));
      // An entry that the scaling itself took to zero is lost whole.
      if (x != 0.f) {
        ++loss.entries;
        loss.add(v != 0.f ? __fdividef(left, fabsf(v)) : 1.f);
      }
    }
    if (d < D) part[(size_t)blockIdx.x * D + d] = loss;
  }
}

// Losses of the columns from those of the blocks: one block per feature, fixed order.
__global__ void __launch_bounds__(128)
column_loss_kernel(const ColumnLoss* __restrict__ part, int nb, int D,
                   ColumnLoss* __restrict__ out) {
  __shared__ ColumnLoss sh[128];
  const int d = blockIdx.x, tid = threadIdx.x;
  ColumnLoss sum{0.f, 0.f, 0u};
  auto merge = [&](const ColumnLoss& c) {
    sum.rest += c.rest;
    sum.add(c.most);
    sum.entries += c.entries;
  };
  for (int b = tid; b < nb; b += 128) merge(part[(size_t)b * D + d]);
  sh[tid] = sum;
  for (int o = 64; o > 0; o >>= 1) {
    __syncthreads();
    if (tid < o) {
      merge(sh[tid + o]);
      sh[tid] = sum;
    }
  }
  if (tid == 0) out[d] = sum;
}

struct F16Rows {
  DeviceBuffer mem;             // hi, lo [N][dp], gscale [D]
  float* gscale = nullptr;      // from G' to G; zero for a column of zeros
  CUtensorMap hi, lo;           // boxes of 64 features x box_rows rows

  // Elements a form may have: beyond its 16 GB the memory is the caller's.
  static constexpr int64_t kMost = (int64_t)1 << 32;

  // Device memory of a form and of its making.
  static int blocks(int num_sms) { return 8 * num_sms; }
  static size_t parts_at(int D) { return (sizeof(unsigned) * (D + 1) + 255) / 256 * 256; }
  static size_t losses_at(int D, int num_sms) {
    return parts_at(D) + (sizeof(ColumnLoss) * (size_t)blocks(num_sms) * D + 255) / 256 * 256;
  }
  static size_t work_bytes(int D, int num_sms) {
    return losses_at(D, num_sms) + sizeof(ColumnLoss) * D;
  }
  static size_t form_bytes(int64_t N, int D, int dp) {
    return 2 * sizeof(__half) * (size_t)N * dp + sizeof(float) * D;
  }
  static size_t bytes(int64_t N, int D, int dp, int num_sms) {
    return N * dp > kMost ? 0 : form_bytes(N, D, dp) + work_bytes(D, num_sms);
  }

  // False if X (or the labels, ym = y - 1/2) does not fit the form: infinities,
  // NaN, exponents that the scaling cannot carry, or a range so wide that hi + lo
  // leaves more than kMostLoss of a column's nonzero entries on average, each relative
  // to the entry; a label so far outside [0, 1] that a residual, below
  // |y - 1/2| + 1/2, could leave FP16's range (R' < 2^16); more than kMost
  // elements, or no memory for it.
  //
  // The average is over entries and not over their squares because which rows count
  // is the residuals' to say: where a fit has a large entry's row right, its residual
  // is zero and the column's gradient is that of the small ones.  2^-23 is what one
  // entry may lose with all of FP16's range above it, so a column without wide range
  // always fits (a normal sample: 2^-25.5 at any length); one entry at 3000 times the
  // others' scale fits, at 10^5 times not, exp(2 normal) fits and exp(3 normal) not.
  // One entry (of 16 or more) may lose any amount: in a sample whose density does not
  // vanish at zero the entry nearest to it, 2^-20 of the others, would otherwise
  // turn one target of 150 away.
  bool prepare(gbm_context* ctx, const float* X, const float* ym, int64_t N, int D, int dp,
               int box_rows) {
    constexpr double kMostLoss = 1.0 / (1 << 23);
    constexpr unsigned kExempt = 16;
    if (N * dp > kMost) return false;
    cudaStream_t s = ctx->stream;
    const int nb = blocks(ctx->num_sms);
    const int64_t chunk = (N + nb - 1) / nb;
    DeviceBuffer buf;
    if (!buf.try_reserve(work_bytes(D, ctx->num_sms)) || !mem.try_reserve(form_bytes(N, D, dp)))
      return false;
    unsigned* mx = buf.as<unsigned>();
    ColumnLoss* part = reinterpret_cast<ColumnLoss*>(buf.as<char>() + parts_at(D));
    ColumnLoss* loss = reinterpret_cast<ColumnLoss*>(buf.as<char>() +
                                                     losses_at(D, ctx->num_sms));
    __half* h = mem.as<__half>();
    __half* l = h + (size_t)N * dp;
    gscale = reinterpret_cast<float*>(l + (size_t)N * dp);
    GBM_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned) * (D + 1), s));
    column_max_kernel<<<nb, 128, 0, s>>>(X, N, D, chunk, mx);
    column_max_kernel<<<nb, 32, 0, s>>>(ym, N, 1, chunk, mx + D);
    f16_pack_kernel<<<nb, 128, 0, s>>>(X, N, D, dp, chunk, mx, h, l, part);
    column_loss_kernel<<<(unsigned)D, 128, 0, s>>>(part, nb, D, loss);
    GBM_CUDA(cudaGetLastError());
    std::vector<unsigned> hmax(D + 1);
    std::vector<ColumnLoss> hloss(D);
    GBM_CUDA(cudaMemcpyAsync(hmax.data(), mx, sizeof(unsigned) * (D + 1), cudaMemcpyDeviceToHost,
                             s));
    GBM_CUDA(cudaMemcpyAsync(hloss.data(), loss, sizeof(ColumnLoss) * D, cudaMemcpyDeviceToHost,
                             s));
    GBM_CUDA(cudaStreamSynchronize(s));
    std::vector<float> gs(D, 0.f);
    constexpr unsigned kLabelTop = 0x3fa00000u;   // 1.25f
    bool fits = hmax[D] <= kLabelTop;
    for (int i = 0; i < D; ++i) {
      if (hmax[i] == 0) continue;
      const int fexp = (int)((hmax[i] >> 23) & 255u) - 127;
      const ColumnLoss& c = hloss[i];
      const double lost = (double)c.rest + (c.entries >= kExempt ? 0.0 : (double)c.most);
      fits = fits && fexp >= -60 && fexp <= 60 && lost <= kMostLoss * (double)c.entries;
      gs[i] = std::ldexp(1.f, fexp - kF16Top - 15);
    }
    if (!fits) {
      mem.release();
      return false;
    }
    GBM_CUDA(cudaMemcpyAsync(gscale, gs.data(), sizeof(float) * D, cudaMemcpyHostToDevice, s));
    GBM_CUDA(cudaStreamSynchronize(s));   // gs ends here
    encode_rows(&hi, h, N, dp, box_rows);
    encode_rows(&lo, l, N, dp, box_rows);
    return true;
  }
};

}  // namespace
}  // namespace gbm
