"""The physics step's branch-free reciprocal and square root (csrc/exact.cuh, Chain) against the IEEE operators, every
binary32 operand of the range they accept, and its division on random and near-midpoint quotients. The kernels are
compiled here from the header; no tolerance: the bits must be equal wherever `ok` stays set."""
import subprocess

import pytest

from warporacer3d_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <stdio.h>
#include "exact.cuh"
using namespace racer;
__device__ unsigned long long bad[4], taken[4];
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__global__ void k_unary() {
  unsigned long long n0 = 0, n1 = 0, b0 = 0, b1 = 0;
  for (unsigned long long u = blockIdx.x * 256ull + threadIdx.x; u < (1ull << 32); u += gridDim.x * 256ull) {
    const float x = __uint_as_float((unsigned)u);
    Chain r;
    const float y = r.rcp(x);
    if (r.ok) ++n0, b0 += !same(y, 1.0f / x);
    Chain q;
    const float g = q.root(x);
    if (q.ok && x <= 1.26765060e30f && !(__float_as_uint(x) >> 31)) ++n1, b1 += !same(g, sqrtf(x));
  }
  atomicAdd(&taken[0], n0), atomicAdd(&bad[0], b0), atomicAdd(&taken[1], n1), atomicAdd(&bad[1], b1);
}
__device__ unsigned mix(unsigned h) {
  h ^= h >> 16, h *= 0x7feb352du, h ^= h >> 15, h *= 0x846ca68bu, h ^= h >> 16;
  return h;
}
// a: random over 2^-60 .. 2^100 and zeros (2), or a hair from a midpoint of b's multiples (3)
__global__ void k_div(int near) {
  unsigned long long n = 0, w = 0;
  for (unsigned k = blockIdx.x * 256 + threadIdx.x; k < (1u << 28); k += gridDim.x * 256) {
    const unsigned h = mix(k * 2 + 1), e = mix(k + 77u);
    const float b = __uint_as_float((h & 0x807fffffu) | ((97u + e % 60u) << 23));
    float a = __uint_as_float((mix(h) & 0x807fffffu) | ((67u + (e >> 8) % 160u) << 23));
    if ((e & 0xffffu) == 7u) a = __uint_as_float(h & 0x80000000u);
    if (near) {  // (q + half an ulp) b rounded, one ulp either way
      const float q = __uint_as_float((mix(h) & 0x7fffffu) | 0x3f800000u);
      a = (float)(((double)q + 5.9604644775390625e-08) * (double)b);
      a = __uint_as_float(__float_as_uint(a) + (e >> 20) % 3u - 1u);
    }
    Chain c;
    const float y = c.rcp(b), d = c.div(a, b, y);
    if (c.ok) ++n, w += !same(d, a / b);
  }
  atomicAdd(&taken[2 + near], n), atomicAdd(&bad[2 + near], w);
}
int main() {
  k_unary<<<1024, 256>>>();
  k_div<<<1024, 256>>>(0);
  k_div<<<1024, 256>>>(1);
  unsigned long long b[4], t[4];
  if (cudaMemcpyFromSymbol(b, bad, sizeof b) != cudaSuccess || cudaMemcpyFromSymbol(t, taken, sizeof t) != cudaSuccess)
    return 2;
  for (int i = 0; i < 4; ++i) printf("%llu %llu\n", t[i], b[i]);
  return 0;
}
"""


def test_chain_operators_are_ieee(tmp_path):
    (tmp_path / "chain.cu").write_text(SOURCE)
    exe = tmp_path / "chain"
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, *build.EXACT, str(tmp_path / "chain.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [[int(v) for v in line.split()] for line in out.splitlines()]
    # rcp: 60 binades of either sign and the two end points; root: 160 positive binades, its end point and zero
    assert rows[0] == [2 * (60 * 2 ** 23 + 1), 0] and rows[1] == [160 * 2 ** 23 + 2, 0]
    for taken, bad in rows[2:]:
        assert bad == 0 and taken > 2 ** 27
