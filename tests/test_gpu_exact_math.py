"""The corrected reciprocal, quotient and square root of exact_math.cuh against the
correctly rounded operations (GPU): near_rcp and near_sqrt at every float of their
ranges, near_div at all dividends' significands over the divisors' edge and random
ones and at random pairs of its whole range.  They start from the hardware's
approximations, so this pins them to the device and the compiler."""
import ctypes
import importlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

build = importlib.import_module("futhark-benchmarks_b200.build")

SOURCE = r"""
#include "exact_math.cuh"
#include <cstdint>
typedef unsigned long long u64;
__device__ __forceinline__ u64 mix(u64 x) {  // a hash of the pair's number
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ __forceinline__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a == 0.0f && b == 0.0f);
}
__device__ __forceinline__ float make(int exponent, uint32_t low) {  // low: sign in bit 23
  return __uint_as_float(((uint32_t)(exponent + 127) << 23) | (low & 0x7fffffu) | ((low & 0x800000u) << 8));
}
// kind 0: near_rcp, 1: near_sqrt, at the floats of the exponents lo .. hi - 1
__global__ void unary(int kind, int lo, int hi, u64* bad) {
  const u64 n = (u64)(hi - lo) << 24;
  u64 mine = 0;
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    const float x = make(lo + (int)(i >> 24), (uint32_t)(i & 0xffffffu));
    if (kind == 0) mine += !same(near_rcp(x), __frcp_rn(x));
    else if (x > 0.0f) mine += !same(near_sqrt(x), __fsqrt_rn(x));
  }
  if (mine) atomicAdd(bad, mine);
}
// every dividend in [1, 2) over divisor number `first` and on: the first and last 64
// significands, then random ones
__global__ void quotients(int divisors, u64* bad) {
  u64 mine = 0;
  for (int d = blockIdx.y; d < divisors; d += gridDim.y) {
    const uint32_t sig = d < 64 ? d : d < 128 ? 0x7fffffu - (d - 64) : (uint32_t)mix(d) & 0x7fffffu;
    const float b = make(0, sig), rb = near_rcp(b);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x) {
      const float a = make(0, i);
      mine += !same(near_div(a, b, rb), __fdiv_rn(a, b));
    }
  }
  if (mine) atomicAdd(bad, mine);
}
// random pairs: |a| in 2^-80 .. 2^80, |b| in 2^-125 .. 2^125, the quotient in 2^-125 .. 2^120
__global__ void pairs(u64 n, u64* bad) {
  u64 mine = 0;
  for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    const u64 r = mix(2 * i), q = mix(2 * i + 1);
    const int ea = (int)(q % 160) - 80, eb = (int)((q >> 20) % 250) - 125;
    if (ea - eb < -124 || ea - eb > 119) continue;
    const float a = make(ea, (uint32_t)r), b = make(eb, (uint32_t)(r >> 32));
    mine += !same(near_div(a, b, near_rcp(b)), __fdiv_rn(a, b));
  }
  if (mine) atomicAdd(bad, mine);
}
extern "C" int check(int kind, u64* differences) {
  u64* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof *d);
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof *d);
  if (e == cudaSuccess) {
    if (kind == 0) unary<<<4096, 256>>>(0, -125, 125, d);
    else if (kind == 1) unary<<<4096, 256>>>(1, -87, 88, d);
    else if (kind == 2) quotients<<<dim3(64, 64), 256>>>(2048, d);
    else pairs<<<4096, 256>>>(1ull << 30, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(differences, d, sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_math")
    (d / "check.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler",
                    "-fPIC", "-shared", "-cudart", "static", "-I", build.CSRC, "-o", str(d / "check.so"),
                    str(d / "check.cu")], check=True)
    return ctypes.CDLL(str(d / "check.so"))


@pytest.mark.parametrize("kind,what", [(0, "near_rcp"), (1, "near_sqrt"), (2, "near_div, all dividends"),
                                       (3, "near_div, random pairs")])
def test_no_difference_from_the_rounded_operation(lib, kind, what):
    bad = ctypes.c_uint64(1)
    assert lib.check(kind, ctypes.byref(bad)) == 0
    assert bad.value == 0, f"{what}: {bad.value} differences"
