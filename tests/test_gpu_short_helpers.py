"""The short square root, reciprocal and quotients against CUDA's correctly rounded intrinsics.

Every float of the square root's and the reciprocal's range; for every significand of the divisor 2,048 dividends,
half of them with a quotient next to a midpoint of two floats, over the exponents that the forces meet and at the ends
of the range; the length of a difference against the general one.
"""

import ctypes
import subprocess

import pytest

from libclsph_gb300.build import ARCH, CSRC, _nvcc

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "clsph_common.cuh"
using namespace clsph;
__device__ __forceinline__ uint32_t mix(uint32_t x) {  // any scrambling of the index will do
  x = (x ^ (x >> 16)) * 0x7feb352du;
  x = (x ^ (x >> 15)) * 0x846ca68bu;
  return x ^ (x >> 16);
}
__device__ __forceinline__ float at_exponent(uint32_t significand, int e) {
  return __uint_as_float(((uint32_t)(e + 127) << 23) | (significand & 0x7FFFFFu));
}
__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

__global__ void roots(uint32_t lo, uint32_t hi, unsigned long long* bad) {
  for (uint64_t b = lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b <= hi; b += (uint64_t)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((uint32_t)b);
    if (!same(sqrt_rn_normal(x), __fsqrt_rn(x))) atomicAdd(bad, 1ull);
  }
}
__global__ void reciprocals(uint32_t lo, uint32_t hi, unsigned long long* bad) {
  for (uint64_t b = lo + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b <= hi; b += (uint64_t)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((uint32_t)b);
    if (!same(rcp_rn_normal(x), __frcp_rn(x))) atomicAdd(bad, 1ull);
  }
}
// divisors: every significand, exponents -24 .. 20; dividends from 2^-100 up, quotients below 2^60
__global__ void quotients(uint32_t dividends, unsigned long long* bad) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < (1u << 23); s += gridDim.x * blockDim.x) {
    for (uint32_t k = 0; k < dividends; ++k) {
      const uint32_t r = mix(s * 2654435761u + k), t = mix(r + k);
      const int eb = (int)(t % 45u) - 24;
      const float b = at_exponent(s, eb), y = rcp_rn_normal(b);
      float a;
      if (k & 1u) {  // a quotient next to a midpoint: the product of b and one, to the nearest float
        const double q = (double)at_exponent(r, 0) + 0x1p-24;
        a = (float)((double)b * q * ((t & 64u) ? 0x1p-70 : (t & 128u) ? 0x1p-20 : 1.0));
      } else {
        int ea = (int)((t >> 8) % 160u) - 100;
        ea = min(ea, eb + 58);
        a = at_exponent(r, ea);
      }
      if (t & 1u) a = -a;
      if (!same(div_rn_normal(a, b, y), __fdiv_rn(a, b))) atomicAdd(bad, 1ull);
    }
    const float b = at_exponent(s, (int)(s % 45u) - 24), y = rcp_rn_normal(b);
    if (div_rn_normal(0.f, b, y) != 0.f || div_rn_normal(-0.f, b, y) != 0.f) atomicAdd(bad, 1ull);
    for (int e = -100; e < -90; ++e)  // the smallest dividends under the largest and the smallest divisors
      for (int big = 0; big < 2; ++big) {
        const float d = at_exponent(s, big ? 20 : -24), a = at_exponent(mix(s + e), e);
        if (!same(div_rn_normal(a, d, rcp_rn_normal(d)), __fdiv_rn(a, d))) atomicAdd(bad, 1ull);
      }
  }
}
__global__ void lengths(uint32_t count, unsigned long long* bad) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint32_t r = mix(i), s = mix(r), t = mix(s);
    auto part = [&](uint32_t x, uint32_t m) {
      const float v = at_exponent(x, (int)(m % 80u) - 59);
      return m & 256u ? -v : m & 512u ? 0.f : v;
    };
    const V3 v = {part(r, t), part(s, t >> 8), part(t, t >> 16)};
    const float exact = xnorm(v), got = near_norm(v);
    if (!same(got, exact >= 0x1p-48f ? exact : 0x1p-48f)) atomicAdd(bad, 1ull);
  }
  const float nan = __uint_as_float(0x7FC00000u), inf = __uint_as_float(0x7F800000u);
  if (near_norm(V3{nan, 0.f, 0.f}) < inf || near_norm(V3{1.f, inf, 0.f}) < 3e38f || near_norm(V3{nan, inf, 1.f}) < inf)
    atomicAdd(bad, 1ull);
}

extern "C" int sweep(int what, unsigned long long* host_bad) {
  unsigned long long* bad = nullptr;
  if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess || cudaMemset(bad, 0, sizeof(*bad)) != cudaSuccess) return 1;
  const dim3 g(152 * 8), b(256);
  if (what == 0) roots<<<g, b>>>(0x0F800000u, 0x7F7FFFFFu, bad);        // 2^-96 .. the largest
  if (what == 1) reciprocals<<<g, b>>>(0x21800000u, 0x5D800000u, bad);  // 2^-60 .. 2^60
  if (what == 2) quotients<<<g, b>>>(2048u, bad);
  if (what == 3) lengths<<<g, b>>>(1u << 28, bad);
  if (cudaGetLastError() != cudaSuccess) return 2;
  const int rc = (int)cudaMemcpy(host_bad, bad, sizeof(*bad), cudaMemcpyDeviceToHost);
  cudaFree(bad);
  return rc;
}
"""


@pytest.fixture(scope="module")
def sweep(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("sweep")
    (d / "sweep.cu").write_text(SOURCE)
    subprocess.run([_nvcc(), *ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", f"-I{CSRC}", "-o",
                    str(d / "sweep.so"), str(d / "sweep.cu")], check=True)
    fn = ctypes.CDLL(str(d / "sweep.so")).sweep

    def run(what):
        bad = ctypes.c_ulonglong(1)
        assert fn(what, ctypes.byref(bad)) == 0
        return bad.value

    return run


@pytest.mark.parametrize("what", ["square roots", "reciprocals", "quotients", "lengths"])
def test_helpers_round_correctly(sweep, what):
    assert sweep(["square roots", "reciprocals", "quotients", "lengths"].index(what)) == 0
