"""The integer form of the decode's double -> float rounding and of its comparisons,
against the hardware's conversion, over every exponent."""
import subprocess

import pytest

from sedona_gpuspatial import _build

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cstdio>
#include "wkb_read.cuh"
using namespace spj::wkb;
// fractions around every tie of the 29 dropped bits, at both ends of the fraction
__device__ double value(uint32_t e, uint32_t i) {
  const uint64_t low[] = {0, 1, 0x0fffffff, 0x10000000, 0x10000001, 0x1fffffff};
  const uint64_t kept[] = {0, 1, 2, 0x3fffff, 0x400000, 0x7ffffe, 0x7fffff, 0x2aaaaa};
  const uint64_t b = (uint64_t)(i / 48 & 1) << 63 | (uint64_t)e << 52 | kept[i / 6 % 8] << 29 | low[i % 6];
  return __longlong_as_double((long long)b);
}
__global__ void check(unsigned* bad) {
  const uint32_t e = blockIdx.x, i = threadIdx.x;
  const double x = value(e, i);
  const float want = __double2float_rn(x), got = f64_to_f32(x);
  const bool same = isnan(want) ? isnan(got) : __float_as_uint(want) == __float_as_uint(got);
  if (!same) atomicAdd(&bad[0], 1u);
  if (isnan(x)) return;
  if (__double_as_longlong(f64_of_key(f64_key(x))) != __double_as_longlong(x)) atomicAdd(&bad[1], 1u);
  for (uint32_t f = 0; f < 2048; f += 23)
    for (uint32_t k = 0; k < 96; k += 7) {
      const double y = value(f, k);
      if (!isnan(y) && x != y && (x < y) != (f64_key(x) < f64_key(y))) atomicAdd(&bad[2], 1u);
    }
}
int main() {
  unsigned *bad, h[3] = {9, 9, 9};
  cudaMalloc(&bad, sizeof h);
  cudaMemset(bad, 0, sizeof h);
  check<<<2048, 96>>>(bad);
  cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
  printf("%u %u %u", h[0], h[1], h[2]);
}
"""


def test_rounding_and_order_on_the_integer_units(tmp_path):
    """Ties, both ends of the float's range, subnormals, overflow, infinities and
    NaN of every exponent."""
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([_build.nvcc(), str(src), "-o", str(exe)] + _build.NVCC_FLAGS, check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    assert out.stdout == "0 0 0"
