// What the tensor-core kernels share: bounded waits that another warp's abort
// ends, error codes, tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "engine.h"
#include "tc_ptx.cuh"

namespace gbm {
namespace {

constexpr uint64_t kWaitLimitNs = 2000000000ull;   // 2 s bound on every device wait

enum TcError : int {
  kTcOk = 0,
  kTcTimeoutTma = 1,
  kTcTimeoutMma = 2,
  kTcTimeoutEpilogue = 3,
};

__device__ __forceinline__ void named_barrier(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Wait that also gives up when another role has already aborted.
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity,
                                              volatile int* abort_flag) {
  if (tc::mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = tc::globaltimer_ns();
  while (true) {
    if (tc::mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (tc::globaltimer_ns() - t0 > kWaitLimitNs) return false;
  }
}

// wait_or_abort by every lane of a warp, with one outcome for the whole warp
// (the .sync.aligned TMEM accesses that follow need a converged warp).
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity,
                                          volatile int* abort_flag) {
  return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    GBM_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                              cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p)
      throw CudaError{cudaErrorNotSupported, "cuTensorMapEncodeTiled entry point"};
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor map over a 16-bit [rows][Dp] matrix: boxes of 64 features x box_rows
// rows, 128-byte swizzle, rows past the end read as zeros.
inline void encode_rows(CUtensorMap* map, void* base, int64_t rows, int Dp, int box_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)Dp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Dp * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw CudaError{cudaErrorInvalidValue, "cuTensorMapEncodeTiled"};
}

}  // namespace
}  // namespace gbm
