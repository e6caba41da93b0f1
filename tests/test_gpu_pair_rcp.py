"""neg_rcp of pair.cuh, on which the packed FP32 arithmetic's equality with the
scalar one rests, against CUDA's correctly rounded reciprocal for every float in
both halves: with the same value in the other half, and with another one (in and
out of the range of the short form)."""
import ctypes
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "flowlb_b200" / "csrc"
SOURCE = r"""
#include "pair.cuh"
using namespace flb;

__device__ bool differs(float got, float x) {
  const float want = -__frcp_rn(x);
  if (want != want) return got == got;
  return __float_as_uint(got) != __float_as_uint(want);
}

// every 32-bit pattern once as the low half; mul 1: the same as the high half,
// another odd number: each pattern once, elsewhere
__global__ void k_check(uint32_t mul, unsigned long long* bad) {
  const uint32_t n = gridDim.x * blockDim.x;
  unsigned long long b = 0;
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 1ull << 32; i += n) {
    const float x = __uint_as_float((uint32_t)i), y = __uint_as_float((uint32_t)i * mul);
    const f2 r = neg_rcp(pack(x, y));
    b += differs(lo(r), x) + differs(hi(r), y);
  }
  if (b) atomicAdd(bad, b);
}

extern "C" int check(uint32_t mul, unsigned long long* bad) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof *d) != cudaSuccess) return 1;
  cudaMemset(d, 0, sizeof *d);
  k_check<<<148 * 8, 256>>>(mul, d);
  const cudaError_t e = cudaMemcpy(bad, d, sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    (d / "rcp.cu").write_text(SOURCE)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", f"-I{CSRC}", str(d / "rcp.cu"), "-o", str(d / "rcp.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "rcp.so"))

    def run(mul):
        bad = ctypes.c_ulonglong()
        assert lib.check(ctypes.c_uint32(mul), ctypes.byref(bad)) == 0
        return bad.value

    return run


@pytest.mark.parametrize("mul", [1, 0x9E3779B1, 0x80000001], ids=["same", "mixed", "opposite"])
def test_every_float(check, mul):
    assert check(mul) == 0
