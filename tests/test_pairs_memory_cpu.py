"""FP32 regressions when there is no memory for the FP16 pairs of X: the target is made
without them, on the CUDA cores.  The constructors run on the host against a fake of
the CUDA runtime whose i-th allocation fails."""
import subprocess

import pytest

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include "logreg_f32.cu"
#include "logreg_simt.cu"
#include "logreg_wide.cu"

extern int fail_at;
size_t held();
namespace gbm {
cudaStream_t& alloc_stream() { static cudaStream_t s = nullptr; return s; }
void set_error(const std::string&) {}
}
// rows features i: the i-th allocation fails (0: none).  Prints the launches of an
// evaluation and the bytes held, or 0 0 where the constructor gave up.
int main(int argc, char** argv) {
  gbm_context ctx;
  ctx.num_sms = 152;
  fail_at = atoi(argv[3]);
  const float* x = reinterpret_cast<const float*>(16);
  try {
    auto t = gbm::make_logreg_simt(&ctx, x, atoi(argv[1]), atoi(argv[2]), x, 1.f);
    printf("%d %zu %d\n", t->launches_per_eval(64), held(), (int)cudaGetLastError());
  } catch (const gbm::CudaError& e) {
    printf("0 0 %d\n", (int)e.err);
  }
}
'''

FAKE = r'''
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>
#include <map>

int fail_at;
static int allocations;
static cudaError_t last = cudaSuccess;
static std::map<void*, size_t> live;
static cudaError_t take(void** p, size_t b) {
  if (++allocations == fail_at) return last = cudaErrorMemoryAllocation;
  *p = malloc(64);
  live[*p] = b;
  return cudaSuccess;
}
static cudaError_t give(void* p) { live.erase(p); free(p); return cudaSuccess; }

static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                       CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }

size_t held() {
  size_t sum = 0;
  for (auto& b : live) sum += b.second;
  return sum;
}

extern "C" {
cudaError_t cudaMalloc(void** p, size_t b) { return take(p, b); }
cudaError_t cudaMallocAsync(void** p, size_t b, cudaStream_t) { return take(p, b); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
  *f = (void*)encode;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset2DAsync(void*, size_t, int, size_t, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind,
                              cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void*, size_t b, cudaMemcpyKind k, cudaStream_t) {
  if (k == cudaMemcpyDeviceToHost) memset(d, 0, b);   // columns of zeros: they fit
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaErrorInvalidValue; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
char __cudaInitModule(void**) { return 1; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
'''


@pytest.fixture(scope='module')
def construct(tmp_path_factory):
  from probability_gb300 import build
  try:
    cc = build.nvcc()
  except RuntimeError as e:
    pytest.skip(str(e))
  d = tmp_path_factory.mktemp('pairs')
  src, fake, exe = str(d / 'pairs.cu'), str(d / 'fake.cpp'), str(d / 'pairs')
  open(src, 'w').write(PROGRAM)
  open(fake, 'w').write(FAKE)
  flags = [f.replace('code=sm_103a', 'code=compute_103a') for f in build._flags() if f != '-O3']
  r = subprocess.run([cc, '-cudart', 'none', src, fake, '-o', exe] + flags, capture_output=True,
                     text=True)
  assert r.returncode == 0, r.stderr

  def run(n, d, i):
    out = subprocess.run([exe, str(n), str(d), str(i)], capture_output=True, text=True, check=True)
    return [int(v) for v in out.stdout.split()]
  return run


def test_up_to_128_features(construct):
  n, d = 5000, 50
  pairs = 4 * n * 64
  launches, held, error = construct(n, d, 0)
  assert (launches, error) == (2, 0) and held > 2 * pairs
  # X, labels and the linear part's two come first: without them there is no target.
  assert [construct(n, d, i)[0] for i in (1, 2, 3, 4)] == [0] * 4
  for i in (5, 6):
    launches, without, error = construct(n, d, i)
    assert (launches, error) == (2, 0)
    assert without == held - pairs - 4 * d


def test_129_to_256_features(construct):
  n, d = 5000, 200
  assert construct(n, d, 0)[0] == 4
  for i in range(1, 6):
    launches, held, error = construct(n, d, i)
    assert (launches, error) == (2, 0)
    assert held == 4 * n * (d + 1)          # X and the labels
