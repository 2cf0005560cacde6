// Element-wise arithmetic of the FP32 logistic-regression kernels: whatever runs a
// chain gets the same bits.
#pragma once
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr float kNegLog2e = -1.4426950408889634f;
constexpr float kLn2f = 0.6931471805599453f;

// -copysign(w, z): magnitude of w with the sign of -z.
__device__ __forceinline__ float neg_copysign_f(float w, float z) {
  return __int_as_float((__float_as_int(w) & 0x7fffffff) |
                        (~__float_as_int(z) & (int)0x80000000));
}

// One row of a chain: r = (y - 1/2) - sign(z) (sigmoid(|z|) - 1/2) and, if the row
// exists, |z| and 1 + e^-|z| into its four rows' sum and product.
__device__ __forceinline__ void f32_residual(float z, float yr, bool valid, float& sabs,
                                             float& prod, float& r) {
  const float a = fabsf(z);
  const float e = tc::ex2_approx(a * kNegLog2e);       // e^-|z|
  const float u1 = 1.f + e;
  if (valid) {
    sabs += a;
    prod *= u1;
  }
  const float w = tc::rcp_approx(u1) - 0.5f;          // sigmoid(|z|) - 1/2
  r = yr + neg_copysign_f(w, z);
}

// The same for two chains, in packed arithmetic (the same roundings).
__device__ __forceinline__ float2 f32_residual2(float2 z, float yr, bool valid, float2& sabs,
                                                float2& prod) {
  const float2 a = make_float2(fabsf(z.x), fabsf(z.y));
  const float2 arg = __fmul2_rn(a, make_float2(kNegLog2e, kNegLog2e));
  const float2 u = __fadd2_rn(make_float2(1.f, 1.f),
                              make_float2(tc::ex2_approx(arg.x), tc::ex2_approx(arg.y)));
  if (valid) {
    sabs = __fadd2_rn(sabs, a);
    prod = __fmul2_rn(prod, u);
  }
  const float2 w = __fadd2_rn(make_float2(tc::rcp_approx(u.x), tc::rcp_approx(u.y)),
                              make_float2(-0.5f, -0.5f));
  return __fadd2_rn(make_float2(yr, yr),
                    make_float2(neg_copysign_f(w.x, z.x), neg_copysign_f(w.y, z.y)));
}

// -(sum |z|/2 + sum ln(1 + e^-|z|)) of four rows.
__device__ __forceinline__ float f32_like(float sabs, float prod) {
  return -fmaf(kLn2f, tc::lg2_approx(prod), 0.5f * sabs);
}

// Kahan: sum += v.
__device__ __forceinline__ void kahan_add(float v, float& sum, float& comp) {
  const float d = v - comp;
  const float t = sum + d;
  comp = (t - sum) - d;
  sum = t;
}

}  // namespace
}  // namespace gbm
