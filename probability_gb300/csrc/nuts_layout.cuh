// Where a chain's vectors live in the NUTS workspace (uniform or ragged
// layout, see NutsDev), for the kernels of samplers.cu and nuts_chain.cu.
#pragma once
#include "samplers.h"

namespace gbm {

__device__ __forceinline__ size_t voff(const NutsDev& w, int c) {
  return w.ragged ? (size_t)w.coff[c] : (size_t)c * w.D;
}
__device__ __forceinline__ int vdim(const NutsDev& w, int c) {
  return w.ragged ? w.cdim[c] : w.D;
}
// Start of U-turn slot i of chain c.
__device__ __forceinline__ size_t soff(const NutsDev& w, int c, int i) {
  return w.ragged ? (size_t)w.coff[c] * w.slots + (size_t)i * w.cdim[c]
                  : ((size_t)c * w.slots + i) * w.D;
}
// Inverse mass of element d of the chain whose vector starts at o (1: identity).
__device__ __forceinline__ float imass(const NutsDev& w, size_t o, int d) {
  return w.inv_mass ? (w.im_per_chain ? w.inv_mass[o + d] : w.inv_mass[d]) : 1.f;
}
__device__ __forceinline__ float eps_of(const float* eps, int per_chain, int c) {
  return per_chain ? eps[c] : eps[0];
}

}  // namespace gbm
