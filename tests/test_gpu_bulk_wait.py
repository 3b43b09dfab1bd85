"""The bounded wait for bulk copies: it reports when it runs out, and a caller that is told
so finds the copies landed."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "plasticity_b200", "csrc")
SOURCE = r"""
#include "bulk_copy.cuh"
constexpr int N = 2048;
__device__ int src[N];
__global__ void fill() { for (int i = threadIdx.x; i < N; i += 32) src[i] = i + 1; }
// copy: start one; else a barrier that nothing completes
__global__ void wait(bool copy, long long polls, long long drain, int* err, int* out) {
  __shared__ __align__(16) int dst[N];
  __shared__ __align__(8) unsigned long long bar;
  const uint32_t b = pfem::bulk_smem(&bar);
  if (threadIdx.x == 0) { pfem::bulk_bar_init(b, 1); pfem::bulk_init_fence(); }
  __syncwarp();
  if (copy && threadIdx.x == 0) { pfem::bulk_expect(b, sizeof(dst)); pfem::bulk_copy(pfem::bulk_smem(dst), src, sizeof(dst), b); }
  const bool ok = pfem::bulk_bar_wait(b, 0, err, polls, drain);
  if (threadIdx.x == 0) out[0] = ok;
  if (copy) {
    int same = 1;
    for (int i = threadIdx.x; i < N; i += 32) same &= dst[i] == i + 1;
    same = __all_sync(0xffffffffu, same);
    if (threadIdx.x == 0) out[1] = same;
  }
}
extern "C" int run(int copy, long long polls, long long drain, int* r) {
  int* d = nullptr;
  cudaMalloc(&d, 12);
  cudaMemset(d, 0, 12);
  fill<<<1, 32>>>();
  wait<<<1, 32>>>(copy != 0, polls, drain, d, d + 1);
  cudaMemcpy(r, d, 12, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("bulk")
    cu, so = d / "wait.cu", d / "wait.so"
    cu.write_text(SOURCE)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-cudart", "static", "-I", CSRC,
                    "-o", str(so), str(cu)], check=True)
    f = C.CDLL(str(so)).run
    f.argtypes = [C.c_int, C.c_longlong, C.c_longlong, C.POINTER(C.c_int)]
    return f


# (a copy is on its way, polls, polls to drain) -> err, waited, landed
@pytest.mark.parametrize("copy,polls,drain,expected", [(1, 1 << 20, 1 << 20, (0, 1, 1)), (1, 0, 1 << 20, (1, 0, 1)),
                                                       (0, 16, 16, (1, 0, 0))])
def test_wait(lib, copy, polls, drain, expected):
    r = (C.c_int * 3)()
    assert lib(copy, polls, drain, r) == 0
    assert tuple(r) == expected
