// Whole NUTS trajectories of hierarchical-normal chains in one launch.
#pragma once
#include <vector>

#include "engine.h"
#include "samplers.h"

namespace gbm {

// Longest vector a chain may have here: four of them are 16 KB of shared
// memory, 13 chains an SM.  Above, a batched leaf has enough work per chain.
constexpr int kChainMaxDim = 1024;

// Reciprocal of the middle of cell i of [1, 2) in 1024 cells.
__host__ __device__ inline float log_table_c(int i) {
  return 1.f / (1.f + ((float)i + 0.5f) / 1024.f);
}
std::vector<double> chain_log_table();   // -log of the above

// Run the chains `models` names: one transition with key f.seed into *single,
// or (single == NULL) f.kmax transitions with keys step_key(f.seed, f.first +
// t) into f's trace, at most max_leaves leapfrog steps a chain.  leaf_max
// (zeroed by the caller): the longest subtree per depth [max_depth] (single),
// or the most leapfrog steps of any chain [1].
void nuts_chain_launch(const NutsDev& w, const FreeDev& f, const ChainModels& models,
                       const float* q, const double* l, const float* g, const NutsOutputs* single,
                       int64_t max_leaves, int32_t* done, int* leaf_max, cudaStream_t s);

}  // namespace gbm
