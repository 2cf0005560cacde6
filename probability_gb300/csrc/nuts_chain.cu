// NUTS transitions of hierarchical-normal chains, one warp per chain, whole
// trajectories in one launch.
//
// A hierarchical-normal gradient is a few hundred operations of the chain's
// own vector, so a batched leaf (compaction, half kick, gradient, leaf
// bookkeeping, each a launch over every chain) is launch latency and passes
// over memory: ~20 us a leaf of an eight-schools batch, 36 us for 4,300
// ragged chains of up to 514 elements.  Nothing couples the chains inside a
// transition (nuts.py:321-1010 only batches them), so here a warp runs its
// chain's trajectories to the end: position, momentum, gradient and momentum
// sum of the growing end stay on the SM (a register a lane up to 32 elements,
// shared memory above), the scalars are warp-uniform registers, and only the
// far end, the candidates and the later U-turn slots are in memory.  A warp that is
// done leaves its place to the next chain's block.
//
// The arithmetic, its order within a lane and the draws are those of the
// batched kernels (samplers.cu, targets_misc.cu, batch.cu), but for the
// prior's log1p, written out below, whose last bit of float64 may differ.
//
// What bounds it: the serial chain of a leaf, and the FP64 pipe (2 lanes a
// clock on an SM: 16 clocks for a warp's instruction), so a leaf's float64
// work is kept to the ~45 instructions that the energies need.  Measured: one
// transition of 256 eight-schools chains 1.18 ms -> 0.15 (kernel 0.14, ~2,000
// clocks a leaf of the longest chain); 4 free-running transitions of 16
// members (4,300 chains, up to 512 groups) 71.5 ms -> 12.3.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "nuts_chain.h"
#include "nuts_layout.cuh"
#include "rng.cuh"

namespace gbm {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kVecs = 4;            // position, momentum, gradient, momentum sum
// Floats of shared memory a warp has at least; what its vectors leave holds
// its first U-turn slots.
constexpr int kWarpFloats = 2048;

struct ChainJob {
  NutsDev w;
  FreeDev f;                 // keys, tables, trace
  const float* q;            // start states, log-densities, gradients
  const double* l;
  const float* g;
  const HierModel* models;
  const int* model_of;       // [C] model of each chain, -1: not run here (NULL: model 0)
  int single;                // one transition with key f.seed, outputs in `out`
  NutsOutputs out;
  long long max_leaves;      // leapfrog steps a chain may take
  int* done;                 // [C] transitions completed, may be NULL
  int* leaf_max;             // single: [max_depth] leaves of the longest subtree; else [1]
};

// Sums of a and of b over the warp: lanes 0-15 reduce a, lanes 16-31 b.  Same
// pairs as two butterflies (warp_sum), at the cost of one.
template <class T>
__device__ __forceinline__ void warp_sum2(T a, T b, int lane, T* sa, T* sb) {
  const bool up = lane >= 16;
  T x = up ? b : a;
  x += __shfl_xor_sync(kAll, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(kAll, x, o);
  *sa = __shfl_sync(kAll, x, 0);
  *sb = __shfl_sync(kAll, x, 16);
}

// log(1 + t^2) to float64 rounding of 1 + log: table lookup and a short series
// (P. T. P. Tang, "Table-driven implementation of the logarithm function in
// IEEE floating-point arithmetic", ACM TOMS 16(4), 1990).  With m the
// mantissa of x = 1 + t^2, i its first 10 fraction bits and c = 1 / (1 + (i +
// 1/2) / 1024) in float32, r = m c - 1 is below 2^-10, log x = e ln 2 - log c +
// r - r^2/2 + r^3 (1/3 - r/4 + r^2/5), and the cubic part is below 2^-31: its
// float32 rounding is below 2^-55.  11 FP64 instructions where the library's
// log1p takes about 60.
__device__ __forceinline__ double log1p_square(float t, const double* neg_log_c) {
  const double td = (double)t;
  const double x = fma(td, td, 1.0);
  const int hi = __double2hiint(x);
  if ((hi & 0x7fffffff) >= 0x7ff00000) return x;   // inf, NaN
  const int i = (hi >> 10) & 1023;
  const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
  const double r = fma(m, (double)log_table_c(i), -1.0);
  const float rf = (float)r;
  const float cubic = rf * rf * rf * fmaf(rf, fmaf(rf, 0.2f, -0.25f), 0.33333334f);
  const double base = fma((double)((hi >> 20) - 1023), 0.6931471805599453, neg_log_c[i]);
  return base + (fma(-0.5 * r, r, r) + (double)cubic);
}

// log_add_exp (common.cuh) without its FP64 comparisons: the same value.
__device__ __forceinline__ double log_add_exp_lean(double x, double y) {
  const double d = x - y;
  const bool xs = !(__double2hiint(d) & 0x80000000);   // x >= y (NaN: either)
  const double l = xs ? x : y;
  // (x - l) + (y - l): NaN for an infinite maximum, else -|x - y|
  const float nd = __double2hiint(l) == 0x7ff00000 ? __int_as_float(0x7fffffff)
                                                   : -fabsf((float)d);
  return l + (double)log1pf(expf(nd));
}

// exp_nonpositive (common.cuh): the power of two added to the exponent bits
// where the result is a normal number.
__device__ __forceinline__ double exp_nonpositive_lean(double x) {
  if (!(x > -690.0)) return exp_nonpositive(x);
  const double t = x * 1.4426950408889634;
  const int n = __double2int_rd(t);
  const double f = (double)exp2f((float)(t - (double)n));
  return __hiloint2double(__double2hiint(f) + (n << 20), __double2loint(f));
}

// A vector of the chain: element lane + 32 k belongs to lane `lane`.  Up to 32
// elements: a register.  Longer: shared memory, in rolled loops (unrolled
// register arrays of 17 elements a lane ran out of instruction cache: 22
// stalls an issue, 21.5 ms where this takes 9.5 for 4,300 chains).
template <bool REG>
struct Vec {
  float r;
  float* s;   // padded to whole warps with zeros
  __device__ __forceinline__ float& at(int lane, int k) { return REG ? r : s[lane + 32 * k]; }
};

template <bool REG>
__device__ __forceinline__ void load_vec(Vec<REG>& v, const float* p, int D, int kc, int lane) {
#pragma unroll 4
  for (int k = 0; k < kc; ++k) v.at(lane, k) = lane + 32 * k < D ? p[lane + 32 * k] : 0.f;
}
template <bool REG>
__device__ __forceinline__ void store_vec(float* p, Vec<REG>& v, int D, int kc, int lane) {
#pragma unroll 4
  for (int k = 0; k < kc; ++k)
    if (lane + 32 * k < D) p[lane + 32 * k] = v.at(lane, k);
}

// One leapfrog gradient of the hierarchical normal (hier_kernel): gradient of
// the log-density at q into g, this lane's share of the likelihood into *lp
// and the rest of the log-density returned.  The likelihood's sums run over
// groups j in lane j % 32; the state's element is j + 2.
template <bool REG>
__device__ __forceinline__ double hier_gradient(const HierModel& m, int J, int lane,
                                                Vec<REG>& q, Vec<REG>& g, float* lp_out) {
  float mu, eta;
  if (REG) {
    mu = __shfl_sync(kAll, q.r, 0);
    eta = __shfl_sync(kAll, q.r, 1);
  } else {
    __syncwarp();
    mu = q.s[0];
    eta = q.s[1];
  }
  const float tau = expf(eta);
  float lp = 0.f, gmu = 0.f, geta = 0.f, gj = 0.f;
  const float zr = REG ? __shfl_sync(kAll, q.r, (lane + 2) & 31) : 0.f;
#pragma unroll 4
  for (int j = lane; j < J; j += 32) {
    const float z = REG ? zr : q.s[j + 2];
    const float s = m.sigma[j];
    const float res = (m.y[j] - (mu + tau * z)) / s;
    const float r = res / s;
    lp += -0.5f * z * z - 0.5f * res * res;
    gmu += r;
    geta += r * z;
    gj = -z + tau * r;
    if (!REG) g.s[j + 2] = gj;
  }
  warp_sum2(gmu, geta, lane, &gmu, &geta);
  const float t = tau / m.tau_scale;
  const double rest = -0.5 * (double)(mu / m.mu_scale) * (double)(mu / m.mu_scale) -
                      log1p_square(t, m.neg_log_c) + (double)eta + m.konst;
  const float g0 = -mu / (m.mu_scale * m.mu_scale) + gmu;
  const float g1 = -2.f * t * t / (1.f + t * t) + 1.f + tau * geta;
  if (REG) {
    g.r = __shfl_sync(kAll, gj, (lane - 2) & 31);
    if (lane == 0) g.r = g0;
    if (lane == 1) g.r = g1;
    if (lane >= J + 2) g.r = 0.f;
  } else {
    if (lane == 0) {
      g.s[0] = g0;
      g.s[1] = g1;
    }
    __syncwarp();
  }
  *lp_out = lp;
  return rest;
}

template <bool REG>
__device__ void run_chain(const ChainJob& job, int c, int lane, float* smem, int smem_floats) {
  const NutsDev& w = job.w;
  const FreeDev& f = job.f;
  const HierModel m = job.models[job.model_of ? job.model_of[c] : 0];
  const int D = vdim(w, c), J = D - 2;
  const int kc = REG ? 1 : (D + 31) >> 5;
  const size_t o = voff(w, c);
  const float eps = eps_of(f.eps_in, f.eps_per_chain, c);
  Vec<REG> q, p, g, cs;
  if (!REG) {
    q.s = smem;
    p.s = q.s + 32 * kc;
    g.s = p.s + 32 * kc;
    cs.s = g.s + 32 * kc;
    smem += kVecs * 32 * kc;
    smem_floats -= kVecs * 32 * kc;
  }
  // Slot i: velocity, and the momentum sum before it.
  const int smem_slots = smem_floats / (2 * D);
  float* const gslot_p = w.slot_p + soff(w, c, 0);
  float* const gslot_cs = w.slot_cs + soff(w, c, 0);
  auto slot_p = [&](int i) { return i < smem_slots ? smem + i * 2 * D : gslot_p + i * D; };
  auto slot_cs = [&](int i) {
    return i < smem_slots ? smem + (i * 2 + 1) * D : gslot_cs + i * D;
  };
  auto im_of = [&](int d) { return d < D ? imass(w, o, d) : 1.f; };
  float* cand_q = w.cand_q + o;   // swapped with the subtree's candidate when it is chosen
  float* cand_g = w.cand_g + o;
  float* sub_q = w.sub_q + o;
  float* sub_g = w.sub_g + o;
  load_vec(q, job.q + o, D, kc, lane);
  load_vec(g, job.g + o, D, kc, lane);
  store_vec(cand_q, q, D, kc, lane);
  store_vec(cand_g, g, D, kc, lane);
  double cand_l = job.l[c];
  long long leaves = 0;
  int t = 0;
  bool budget = true;
  for (; t < f.kmax; ++t) {
    const uint2 key = job.single ? f.seed : step_key(f.seed, f.first + (uint32_t)t);
    // ---- trajectory start (nuts.py:512-539): momentum, both ends ----
    const uint32_t msite = draw_site(kDrawMomentum, 0, 0);
    float kin_l = 0.f;
#pragma unroll 1
    for (int k = 0; k < kc; ++k) {
      const int d = lane + 32 * k;
      float pd = 0.f;
      if (d < D) {
        const float im = imass(w, o, d);
        pd = w.inv_mass ? draw_normal(key, msite, (uint32_t)(o + d)) / sqrtf(im)
                        : draw_normal(key, msite, (uint32_t)(o + d));
        kin_l = fmaf(pd * im, pd, kin_l);
      }
      p.at(lane, k) = pd;
    }
    store_vec(w.end_q[0] + o, q, D, kc, lane);
    store_vec(w.end_p[0] + o, p, D, kc, lane);
    store_vec(w.end_g[0] + o, g, D, kc, lane);
    store_vec(w.mom_sum + o, p, D, kc, lane);
    const double e0 = cand_l - 0.5 * warp_sum((double)kin_l);
    double cand_e = e0, cand_w = 0.0, eds = 0.0;
    int lf = 0, depth = 0;
    bool accepted = false, not_div = true, cont = true;
    int side = 1;   // the end held here; the other one is in memory
    // Lane d holds the direction and the tree-level uniform of depth d, and
    // below the uniform of leaf 32 i + lane: one Philox for 32 draws.
    const int fwd_l = draw_direction(key, (uint32_t)lane, (uint32_t)c);
    const float tree_l = (float)log1m_uniform(
        draw_uniform(key, draw_site(kDrawTreeUniform, lane, 0), (uint32_t)c));
    while (true) {
      // ---- one doubling: a subtree of up to 2^depth leaves ----
      const int fwd = __shfl_sync(kAll, fwd_l, depth);
      if (fwd != side) {
        store_vec(w.end_q[side] + o, q, D, kc, lane);
        store_vec(w.end_p[side] + o, p, D, kc, lane);
        store_vec(w.end_g[side] + o, g, D, kc, lane);
        side = fwd;
        load_vec(q, w.end_q[side] + o, D, kc, lane);
        load_vec(p, w.end_p[side] + o, D, kc, lane);
        load_vec(g, w.end_g[side] + o, D, kc, lane);
      }
      const float e = (side ? 1.f : -1.f) * eps;
      const float he = 0.5f * e;
      double sub_w = -INFINITY, sub_eds = 0.0, sub_l = 0.0, sub_e = 0.0;
      int sub_lf = 0;
      bool sub_cont = true, sub_not_div = not_div;
#pragma unroll 4
      for (int k = 0; k < kc; ++k) cs.at(lane, k) = 0.f;
      float leaf_l = 0.f;
      for (int leaf = 0; leaf < (1 << depth) && sub_cont; ++leaf) {
        if (leaves == job.max_leaves) {
          budget = false;
          break;
        }
        ++leaves;
        const int wslot = f.wtab[leaf], r0 = f.rlo[leaf], r1 = f.rhi[leaf];
        if ((leaf & 31) == 0)
          leaf_l = (float)log1m_uniform(draw_uniform(
              key, draw_site(kDrawLeafUniform, depth, leaf + lane), (uint32_t)c));
        // half kick and drift (leapfrog_integrator.py:280-286, :330-334)
#pragma unroll 4
        for (int k = 0; k < kc; ++k) {
          const float ph = p.at(lane, k) + he * g.at(lane, k);
          p.at(lane, k) = ph;
          q.at(lane, k) = q.at(lane, k) + e * (ph * im_of(lane + 32 * k));
        }
        float lp;
        const double rest = hier_gradient<REG>(m, J, lane, q, g, &lp);
        // second half of the kick, momentum sum, U-turn slot (nuts.py:793-946)
        float kl = 0.f;
        float* const wp = slot_p(wslot < 0 ? 0 : wslot);
        float* const wc = slot_cs(wslot < 0 ? 0 : wslot);
#pragma unroll 4
        for (int k = 0; k < kc; ++k) {
          const int d = lane + 32 * k;
          const float gd = g.at(lane, k), csp = cs.at(lane, k);
          const float p2 = (p.at(lane, k) + e * gd) - he * gd;
          const float im = im_of(d);
          p.at(lane, k) = p2;
          if (wslot >= 0 && d < D) {
            wp[d] = p2 * im;
            wc[d] = csp;
          }
          cs.at(lane, k) = csp + p2;
          kl = fmaf(p2 * im, p2, kl);
        }
        double lpd, kin;
        warp_sum2((double)lp, (double)kl, lane, &lpd, &kin);
        bool no_uturn = true;
#pragma unroll 1
        for (int i = r0; i < r1; ++i) {
          float dl = 0.f, dr = 0.f;
          const float* sp = slot_p(i);
          const float* sc = slot_cs(i);
#pragma unroll 4
          for (int k = 0; k < kc; ++k) {
            const int d = lane + 32 * k;
            if (d < D) {
              const float diff = cs.at(lane, k) - sc[d];
              dl = fmaf(diff, sp[d], dl);
              dr = fmaf(diff, p.at(lane, k) * im_of(d), dr);
            }
          }
          warp_sum2(dl, dr, lane, &dl, &dr);
          no_uturn = no_uturn && (dl >= 0.f) && (dr >= 0.f);
        }
        const double l2 = lpd + rest;
        double energy = l2 - 0.5 * kin;
        if (isnan(energy)) energy = -INFINITY;
        const double de = energy - e0;
        const bool leaf_ok = -de < f.max_energy_diff;
        const double wsum = log_add_exp_lean(sub_w, de);
        const double thresh = de - wsum;
        if ((double)__shfl_sync(kAll, leaf_l, leaf & 31) <= thresh) {
          store_vec(sub_q, q, D, kc, lane);
          store_vec(sub_g, g, D, kc, lane);
          sub_l = l2;
          sub_e = energy;
        }
        sub_w = wsum;
        if (leaf_ok) sub_eds += exp_nonpositive_lean(fmin(de, 0.0));
        ++sub_lf;
        if (!leaf_ok) sub_not_div = false;
        sub_cont = leaf_ok && no_uturn;
      }
      if (!budget) break;
      if (job.single && lane == 0) atomicMax(job.leaf_max + depth, sub_lf);
      // ---- tree level (nuts.py:597-711) ----
      const double tree_w = sub_cont ? sub_w : -INFINITY;
      const double wsum = log_add_exp(tree_w, cand_w);
      double thresh = tree_w - cand_w;
      if (isnan(thresh)) thresh = 0.0;
      const bool choose = ((double)__shfl_sync(kAll, tree_l, depth) <= thresh) && sub_cont;
      float dl = 0.f, dr = 0.f;
      const float* far = w.end_p[side ^ 1] + o;
#pragma unroll 4
      for (int k = 0; k < kc; ++k) {
        const int d = lane + 32 * k;
        if (d < D) {
          const float ms = w.mom_sum[o + d] + cs.at(lane, k);
          w.mom_sum[o + d] = ms;
          const float im = imass(w, o, d), near = p.at(lane, k), other = far[d];
          dl = fmaf(ms, (side ? other : near) * im, dl);
          dr = fmaf(ms, (side ? near : other) * im, dr);
        }
      }
      warp_sum2(dl, dr, lane, &dl, &dr);
      if (choose) {
        float* x = cand_q; cand_q = sub_q; sub_q = x;
        x = cand_g; cand_g = sub_g; sub_g = x;
        cand_l = sub_l;
        cand_e = sub_e;
        accepted = true;
      }
      cand_w = wsum;
      eds += sub_eds;
      lf += sub_lf;
      cont = sub_cont && (dl >= 0.f && dr >= 0.f);
      not_div = sub_not_div;
      ++depth;
      if (!cont || depth >= f.max_depth) break;
    }
    if (!budget) break;
    // ---- the transition's results (nuts.py:424-441) ----
    load_vec(q, cand_q, D, kc, lane);
    load_vec(g, cand_g, D, kc, lane);
    const size_t row = (size_t)t * w.C + c;
    const double lar = log(eds / (double)lf);
    if (job.single) {
      const NutsOutputs& out = job.out;
      if (out.state) store_vec(out.state + o, q, D, kc, lane);
      if (out.grads) store_vec(out.grads + o, g, D, kc, lane);
      if (lane == 0) {
        if (out.target_log_prob) out.target_log_prob[c] = cand_l;
        if (out.log_accept_ratio) out.log_accept_ratio[c] = lar;
        if (out.leapfrogs_taken) out.leapfrogs_taken[c] = lf;
        if (out.is_accepted) out.is_accepted[c] = accepted;
        if (out.reach_max_depth) out.reach_max_depth[c] = cont;
        if (out.has_divergence) out.has_divergence[c] = !not_div;
        if (out.energy) out.energy[c] = cand_e;
        if (out.tree_depth) out.tree_depth[c] = depth;
      }
    } else {
      if (f.tr_state) store_vec(f.tr_state + (size_t)t * f.tr_estride + o, q, D, kc, lane);
      if (lane == 0) {
        if (f.tr_logp) f.tr_logp[row] = cand_l;
        if (f.tr_lar) f.tr_lar[row] = lar;
        if (f.tr_lf) f.tr_lf[row] = lf;
        if (f.tr_acc) f.tr_acc[row] = accepted;
        if (f.tr_div) f.tr_div[row] = !not_div;
      }
      if (f.mom_mean) {   // as moments_update_kernel, with this chain's draw count
        const double inv_count = 1.0 / (double)(f.mom_base + t + 1);
#pragma unroll 1
        for (int d = lane, k = 0; d < D; d += 32, ++k) {
          const double v = (double)q.at(lane, k);
          const double delta = v - f.mom_mean[o + d];
          const double mnew = f.mom_mean[o + d] + delta * inv_count;
          f.mom_mean[o + d] = mnew;
          f.mom_m2[o + d] += delta * (v - mnew);
        }
      }
    }
  }
  // sample_chain picks the final state up from the workspace.
  if (cand_q != w.cand_q + o) {
    load_vec(q, cand_q, D, kc, lane);
    load_vec(g, cand_g, D, kc, lane);
    store_vec(w.cand_q + o, q, D, kc, lane);
    store_vec(w.cand_g + o, g, D, kc, lane);
  }
  if (lane == 0) {
    w.cand_l[c] = cand_l;
    if (job.done) job.done[c] = t;
    if (!job.single)
      atomicMax(job.leaf_max, (int)(leaves < 0x7fffffff ? leaves : 0x7fffffff));
  }
}

// One warp per block, one chain per block: an SM's place is taken by the next
// chain as soon as one is done.  REG: every chain has at most 32 elements.
template <bool REG>
__global__ void __launch_bounds__(32, 20) nuts_chain_kernel(ChainJob job, int smem_floats) {
  extern __shared__ __align__(16) float chain_smem[];
  const int c = blockIdx.x, lane = threadIdx.x;
  if (job.model_of && job.model_of[c] < 0) return;
  run_chain<REG>(job, c, lane, chain_smem, smem_floats);
}

}  // namespace

void nuts_chain_launch(const NutsDev& w, const FreeDev& f, const ChainModels& models,
                       const float* q, const double* l, const float* g, const NutsOutputs* single,
                       int64_t max_leaves, int32_t* done, int* leaf_max, cudaStream_t s) {
  ChainJob job{};
  job.w = w;
  job.f = f;
  job.q = q;
  job.l = l;
  job.g = g;
  job.models = models.models;
  job.model_of = models.model_of;
  job.single = single != nullptr;
  if (single) job.out = *single;
  job.max_leaves = max_leaves;
  job.done = done;
  job.leaf_max = leaf_max;
  const int pad = (models.max_dim + 31) / 32 * 32;
  const int vecs = models.max_dim <= 32 ? 0 : kVecs * pad;
  const int floats = std::max(kWarpFloats, vecs);
  const size_t bytes = sizeof(float) * (size_t)floats;
  if (vecs == 0) nuts_chain_kernel<true><<<w.C, 32, bytes, s>>>(job, floats);
  else nuts_chain_kernel<false><<<w.C, 32, bytes, s>>>(job, floats);
  GBM_CUDA(cudaGetLastError());
}

// -log c of log1p_square's table, for the models' upload.
std::vector<double> chain_log_table() {
  std::vector<double> t(1024);
  for (int i = 0; i < 1024; ++i) t[i] = -std::log((double)log_table_c(i));
  return t;
}

}  // namespace gbm
