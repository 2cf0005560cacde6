// One tile of a multivariate normal's two triangular products, shared by the
// single target (targets_misc.cu) and the ragged batch (batch.cu).
//
//   PHASE 0:  U[c][o] = sum_{k <= o} (x_c[k] - loc[k]) L^-1[o][k]
//             part[c][b] = sum of U[c][o]^2 over the 32 outputs of block b
//   PHASE 1:  G[c][o] = -sum_{k >= o} U_c[k] L^-1[k][o]; the last output block
//             also writes logp = -1/2 sum_b part[c][b] + log_norm.
//
// A tile is CT chains x OB outputs over every k that reaches them.  The factor
// is kept twice, transposed for phase 0 and as it is for phase 1, zero outside
// its triangle and padded to multiples of 64, so that both phases read rows of
// consecutive outputs by 16-byte asynchronous copies.  The chains' values (which
// may begin anywhere) are copied 4 bytes at a time as they lie, and the thread
// that copied a value moves it, less loc, to [k][chain] order when it has landed.
// A thread holds 4 chains x RO outputs and multiplies two outputs an instruction
// (fma.rn.f32x2); a warp is 4 x 8 threads.
//
// An output of phase 0 is one chain of FMAs in ascending k, so the log-density
// does not depend on the tile; phase 1 cuts k into KG stretches of whole 32s,
// each with its own threads, and adds their sums in order.  Neither depends on
// CT or on which chains are active: those are a matter of speed only.
//
// What bounds it: where tiles fill the machine, shared loads (a warp's 16-byte
// load takes the SM's port for four clocks: 8 clocks for the 16 FMAs of a 4 x 4
// thread, 12 for the 32 of a 4 x 8 one); where they do not, the chain of k, 60
// clocks a step with one warp on each SM quarter (issue, and shared-memory latency
// that a lone warp cannot hide).  One tile of 64 x 64 a CTA with two stages filled
// through registers took 105.  Measured, whole evaluations: 777 x 350 chains 146 us
// before, 52 so; 2048 x 512 446 and 175; 300 x 300 70 and 29; the ragged batch
// below 521 and 207.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace gbm {

constexpr int kMvnPad = 64;      // the factor's sides are padded to this
constexpr int kMvnPart = 32;     // outputs whose squares are summed together

// L^-1 of one normal as the tiles read it.
struct MvnFactor {
  int dim, pad;                  // D, and D rounded up to kMvnPad
  const float* loc;              // [D]
  const float* upper;            // [pad][pad]: [k][o] = L^-1[o][k]  (phase 0)
  const float* lower;            // [pad][pad]: [k][o] = L^-1[k][o]  (phase 1)
  double log_norm;
};

__host__ __device__ inline int mvn_pad(int64_t d) {
  return (int)((d + kMvnPad - 1) / kMvnPad * kMvnPad);
}
__host__ __device__ inline int mvn_parts(int64_t d) {
  return (int)((d + kMvnPart - 1) / kMvnPart);
}
inline size_t mvn_factor_bytes(int64_t d) {
  return 2 * sizeof(float) * (size_t)mvn_pad(d) * mvn_pad(d);
}

namespace {
// L^-1 [D][D] -> its two padded forms.
__global__ void mvn_pack_kernel(const float* __restrict__ linv, int D, int pad,
                                float* __restrict__ upper, float* __restrict__ lower) {
  __shared__ float t[32][33];
  const int k0 = blockIdx.x * 32, o0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int row = o0 + r, col = k0 + threadIdx.x;
    const float v = (row < D && col <= row) ? linv[(size_t)row * D + col] : 0.f;
    lower[(size_t)row * pad + col] = v;
    t[r][threadIdx.x] = v;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y)
    upper[(size_t)(k0 + r) * pad + o0 + threadIdx.x] = t[threadIdx.x][r];
}

// Lays the factor out in `mem` (mvn_factor_bytes(d), device).
inline MvnFactor mvn_factor(const float* linv, const float* loc, int64_t d, double log_norm,
                            float* mem, cudaStream_t s) {
  const int pad = mvn_pad(d);
  MvnFactor f{(int)d, pad, loc, mem, mem + (size_t)pad * pad, log_norm};
  mvn_pack_kernel<<<dim3(pad / 32, pad / 32), dim3(32, 8), 0, s>>>(
      linv, (int)d, pad, mem, mem + (size_t)pad * pad);
  GBM_CUDA(cudaGetLastError());
  return f;
}

template <int CT, int OB, int KG>
struct alignas(16) MvnSmem {
  // Steps of k of a chunk, and chunks in flight or in use: both as large as four
  // CTAs on an SM leave room for.
  static constexpr int kRows = CT == 64 ? 16 : 32;
  static constexpr int kRing = CT == 64 ? 4 : 3;
  struct Group {
    float Bs[kRing][kRows][OB];    // [stage][k][output]
    float raw[kRing][CT][kRows];   // [stage][chain][k], as they lie
    float As[2][kRows][CT + 4];    // [stage][k][chain]
  } group[KG];
  double red[OB / kMvnPart][CT];
  // Per chain of the tile: element offset of its input and output vector,
  // offset of its partials, index of its log-density.
  long long in[CT], out[CT], part[CT];
  int id[CT];
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
// Four bytes, or zero without a read.
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool held) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(held ? 4 : 0)
               : "memory");
}

__device__ __forceinline__ void group_barrier(int group, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}

// Outputs [o0, o0 + OB) of the tile's nc chains, whose offsets the caller has
// put into sm (not yet visible to all threads).  KG groups of threads share the
// chunks of k between them and add their sums at the end, in order (phase 1:
// phase 0 keeps one ascending chain).
template <int PHASE, int CT, int OB, int RC, int RO, int KG>
__device__ __forceinline__ void mvn_tile(const MvnFactor f, int nc, int o0,
                                         const float* __restrict__ X, float* __restrict__ out,
                                         double* __restrict__ part, double* __restrict__ logp,
                                         MvnSmem<CT, OB, KG>& sm) {
  using Smem = MvnSmem<CT, OB, KG>;
  constexpr int kThreads = CT / RC * (OB / RO);   // of a group
  constexpr int kRows = Smem::kRows, kRing = Smem::kRing, kStep = kThreads / kRows;
  constexpr int kAhead = RO == 4 ? 4 : 2;         // steps of k whose fragments load together
  constexpr int kWarpsO = OB / (8 * RO);          // warps beside each other in outputs
  constexpr int AL = kRows * CT / kThreads, BL = kRows * OB / 4 / kThreads;
  static_assert(RC == 4 && (RO == 4 || RO == 8), "thread tile");
  static_assert(PHASE == 1 || KG == 1, "phase 0 is one chain of k");
  static_assert(AL * kThreads == kRows * CT && BL * kThreads * 4 == kRows * OB, "tile loads");
  const int group = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
  const int warp = tid >> 5, lane = tid & 31;
  typename Smem::Group& gs = sm.group[group];
  const int wo = warp % kWarpsO, wc = warp / kWarpsO;
  const int a_at = wc * 4 * RC + (lane >> 3) * RC;          // first chain of this thread
  const int b_at = wo * 8 * RO + (lane & 7) * 4;            // first output (and 32 on)
  const int D = f.dim;
  const float* B = (PHASE == 0 ? f.upper : f.lower) + o0;
  // This group's stretch of k, in units of 32 whatever the chunk.
  const int k_first = PHASE == 0 ? 0 : o0, k_last = PHASE == 0 ? min(D, o0 + OB) : D;
  const int units = (k_last - k_first + 31) / 32;
  const int k_begin = k_first + group * units / KG * 32;
  const int k_end = min(k_last, k_first + (group + 1) * units / KG * 32);
  const int chunks = k_end > k_begin ? (k_end - k_begin + kRows - 1) / kRows : 0;
  float2 acc[RC][RO / 2];
#pragma unroll
  for (int i = 0; i < RC; ++i)
#pragma unroll
    for (int j = 0; j < RO / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
  // This thread's share of a chunk: k index ak of chains ac, ac + kThreads /
  // kRows, ... and BL vectors of the factor.
  const int ak = tid % kRows, ac = tid / kRows;
  __syncthreads();   // the caller's offsets
  const float* row[AL];
#pragma unroll
  for (int r = 0; r < AL; ++r) {
    const int cc = ac + r * kStep;
    row[r] = X + (cc < nc ? sm.in[cc] : sm.in[0]) + k_begin + ak;
  }
  auto copy = [&](int ch) {
    if (ch < chunks) {
      const int st = ch % kRing, k0 = ch * kRows;
      const bool mine = k_begin + k0 + ak < D;
#pragma unroll
      for (int r = 0; r < AL; ++r) {
        const int cc = ac + r * kStep;
        const bool held = mine && cc < nc;
        cp_async4(&gs.raw[st][cc][ak], held ? row[r] + k0 : X, held);
      }
#pragma unroll
      for (int r = 0; r < BL; ++r) {
        const int i = tid + r * kThreads, k = i / (OB / 4), o = i % (OB / 4) * 4;
        cp_async16(&gs.Bs[st][k][o], B + (size_t)(k_begin + k0 + k) * f.pad + o);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto loc_of = [&](int ch) {
    const int k = k_begin + ch * kRows + ak;
    return PHASE == 0 && k < D ? f.loc[k] : 0.f;
  };
  auto turn = [&](int ch, float loc) {   // this thread's values of chunk ch
#pragma unroll
    for (int r = 0; r < AL; ++r) {
      const int cc = ac + r * kStep;
      const float v = gs.raw[ch % kRing][cc][ak];
      const float w = PHASE == 0 ? (cc < nc ? v - loc : 0.f) : v;
      gs.As[ch & 1][ak][cc] = w;
    }
  };
#pragma unroll
  for (int ch = 0; ch < kRing - 1; ++ch) copy(ch);
  float loc = loc_of(0), loc_next = loc_of(1);
  asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
  if (chunks > 0) turn(0, loc);
  group_barrier(group, kThreads);
  for (int ch = 0; ch < chunks; ++ch) {
    const int st = ch & 1, sb = ch % kRing;
    // The next chunk's copies have landed; the stages of the last one are free.
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 3) : "memory");
    loc = loc_next;
    loc_next = loc_of(ch + 2);
    if (ch + 1 < chunks) turn(ch + 1, loc);
    copy(ch + kRing - 1);
    // The next steps' fragments load while these ones' FMAs issue.
    const float* ap = &gs.As[st][0][a_at];
    const float* bp = &gs.Bs[sb][0][b_at];
    float4 av[kAhead], bv[kAhead][RO / 4], an[kAhead], bn[kAhead][RO / 4];
    auto fragments = [&](int k0, float4(&x)[kAhead], float4(&y)[kAhead][RO / 4]) {
#pragma unroll
      for (int g = 0; g < kAhead; ++g) {
        x[g] = *reinterpret_cast<const float4*>(ap + (k0 + g) * (CT + 4));
#pragma unroll
        for (int h = 0; h < RO / 4; ++h)
          y[g][h] = *reinterpret_cast<const float4*>(bp + (k0 + g) * OB + 32 * h);
      }
    };
    fragments(0, av, bv);
#pragma unroll
    for (int kk = 0; kk < kRows; kk += kAhead) {
      if (kk + kAhead < kRows) fragments(kk + kAhead, an, bn);
#pragma unroll
      for (int g = 0; g < kAhead; ++g) {
        const float aa[4] = {av[g].x, av[g].y, av[g].z, av[g].w};
#pragma unroll
        for (int h = 0; h < RO / 4; ++h)
#pragma unroll
          for (int i = 0; i < RC; ++i) {
            const float2 a2 = make_float2(aa[i], aa[i]);
            acc[i][2 * h] = __ffma2_rn(a2, make_float2(bv[g][h].x, bv[g][h].y), acc[i][2 * h]);
            acc[i][2 * h + 1] =
                __ffma2_rn(a2, make_float2(bv[g][h].z, bv[g][h].w), acc[i][2 * h + 1]);
          }
      }
#pragma unroll
      for (int g = 0; g < kAhead; ++g) {
        av[g] = an[g];
#pragma unroll
        for (int h = 0; h < RO / 4; ++h) bv[g][h] = bn[g][h];
      }
    }
    // Chunk ch + 1 is complete, the stages of this one are free.
    group_barrier(group, kThreads);
  }
  if (KG > 1) {
    // The groups' sums go where their chunks were, and are added from there.
    float* mine = &gs.raw[0][0][0];
    static_assert(Smem::kRing * CT * kRows >= CT * OB, "a group's sums fit its stages");
#pragma unroll
    for (int i = 0; i < RC; ++i)
#pragma unroll
      for (int h = 0; h < RO / 4; ++h)
        *reinterpret_cast<float4*>(mine + (a_at + i) * OB + b_at + 32 * h) =
            make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
    __syncthreads();
    for (int i = threadIdx.x; i < CT * OB; i += KG * kThreads) {
      const int cc = i / OB, o = o0 + i % OB;
      float v = (&sm.group[0].raw[0][0][0])[i];
#pragma unroll
      for (int g = 1; g < KG; ++g) v += (&sm.group[g].raw[0][0][0])[i];
      if (cc < nc && o < D) out[sm.out[cc] + o] = -v;
    }
  } else {
#pragma unroll
    for (int i = 0; i < RC; ++i) {
      const int cc = a_at + i;
#pragma unroll
      for (int h = 0; h < RO / 4; ++h) {
        const float v[4] = {acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x,
                            acc[i][2 * h + 1].y};
        double sq = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int o = o0 + b_at + 32 * h + j;
          if (cc < nc && o < D) {
            out[sm.out[cc] + o] = PHASE == 0 ? v[j] : -v[j];
            sq += (double)v[j] * (double)v[j];
          }
        }
        if (PHASE == 0) {
#pragma unroll
          for (int m = 1; m < 8; m <<= 1) sq += __shfl_xor_sync(~0u, sq, m);
          if ((lane & 7) == 0) sm.red[wo + h][cc] = sq;
        }
      }
    }
  }
  if (PHASE == 0) {
    __syncthreads();
    for (int i = threadIdx.x; i < CT * (OB / kMvnPart); i += KG * kThreads) {
      const int cc = i % CT, b = o0 / kMvnPart + i / CT;
      if (cc < nc && b * kMvnPart < D) part[sm.part[cc] + b] = sm.red[i / CT][cc];
    }
  } else if (o0 + OB >= D && (int)threadIdx.x < nc) {   // the shortest tile of its chains
    const double* p = part + sm.part[threadIdx.x];
    const int np = mvn_parts(D);
    double s = 0.0;
#pragma unroll 8
    for (int b = 0; b < np; ++b) s += p[b];
    logp[sm.id[threadIdx.x]] = -0.5 * s + f.log_norm;   // -1/2 |L^-1 (x - loc)|^2 + normaliser
  }
}

}  // namespace

}  // namespace gbm
