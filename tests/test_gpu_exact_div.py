"""csrc/exact_div.cuh on the device: the reciprocal's seed stays within the
2^-18 that the method needs, for every significand the seed can tell apart
(it reads the upper 32 bits: each is tried with the lowest and the highest
lower half), and quotients and reciprocals are the bits of the device's own
division on the operand classes of tests/test_exact_div.py."""
import os
import subprocess

import pytest

from harm_finalwham_b200.build import ARCH
from tests.test_exact_div import CSRC

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "exact_div.cuh"
#include <cstdio>
#include <cstdlib>
using namespace hg;
__device__ uint64_t next(uint64_t &s) {  // splitmix64
  uint64_t z = (s += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ double make(uint64_t m, int e, bool neg) {
  return __longlong_as_double((long long)((uint64_t)(1023 + e) << 52 | (m & ((1ull << 52) - 1)) | (uint64_t)neg << 63));
}
__device__ bool bits(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y) || (x != x && y != y);
}
// out[0]: seeds off by 2^-18 or more
__global__ void seeds(unsigned long long *out) {
  const uint64_t top = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;  // 2^20 upper significand parts
  const int es[] = {-200, -1, 0, 1, 199};
  for (int q = 0; q < 5; q++)
    for (int low = 0; low < 2; low++) {
      const double b = make(top << 32 | (low ? 0xffffffffull : 0ull), es[q], false);
      if (!(fabs(fma(-b, rcp_seed(b), 1.0)) < 0x1p-18)) atomicAdd(out, 1ull);
    }
}
// out[0]: quotients or reciprocals other than the division's; out[1]: divisors in range
__global__ void quotients(int kind, unsigned long long *out) {
  uint64_t s = (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 1000003ull + kind;
  unsigned bad = 0, used = 0;
  for (int n = 0; n < 64; n++) {
    uint64_t ma = next(s), mb = next(s);
    int ea = (int)(next(s) % 60) - 30, eb = (int)(next(s) % 60) - 30;
    if (kind == 1) mb = ~(next(s) % 64);
    if (kind == 2) mb = next(s) % 64;
    if (kind == 3) { ma = ~(next(s) % 64); mb = ~(next(s) % 1024); }
    if (kind == 5) { ea = (int)(next(s) % 1400) - 700; eb = (int)(next(s) % 400) - 200; }
    double b = make(mb, eb, false), a = make(ma, ea, next(s) & 1);
    if (kind == 4) a = nextafter(make(next(s), 0, false) * b, next(s) & 1 ? 1e300 : 0.0);  // quotient near a middle
    double num[3] = {a, -a, a}, q[3];
    if (kind == 6) {
      const double odd[] = {0.0, -0.0, 4e-324, -1e-310, 1e-250, 1e300, INFINITY, -INFINITY, NAN, 1.0};
      const double den[] = {b, 1e-100, 1e100, 5e-324, INFINITY, NAN, make(~0ull, eb, false), 0.0};
      num[1] = odd[next(s) % 10];
      num[2] = odd[next(s) % 10];
      b = den[next(s) % 8];
    }
    if (kind == 7) {
      b = -b;
      if (next(s) % 3 == 0) num[next(s) % 3] = next(s) & 1 ? 0.0 : -0.0;
    }
    const Divisor<double> d = make_divisor(b);
    if (d.ok) {
      used++;
      bad += !bits(d.y, 1.0 / b);
    }
    div_n<3>(num, d, q);
    for (int i = 0; i < 3; i++) bad += !bits(q[i], num[i] / b);
  }
  if (bad) atomicAdd(out, (unsigned long long)bad);
  atomicAdd(out + 1, (unsigned long long)used);
}
int main(int argc, char **argv) {
  const int kind = atoi(argv[1]);
  unsigned long long *out, h[2];
  if (cudaMalloc(&out, sizeof(h)) || cudaMemset(out, 0, sizeof(h))) return 1;
  if (kind < 0) seeds<<<4096, 256>>>(out);
  else quotients<<<1024, 256>>>(kind, out);
  if (cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost)) return 1;
  printf("%llu %llu\n", h[0], h[1]);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("gpu_exact_div")
    (d / "t.cu").write_text(SOURCE)
    exe = str(d / "t")
    subprocess.run([os.environ.get("NVCC", "nvcc")] + ARCH + ["-O3", "-std=c++17", "-fmad=false", "-I", CSRC, "-o", exe,
                    str(d / "t.cu")], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("kind", range(-1, 8))
def test_the_devices_quotients_are_its_divisions_bits(program, kind):
    out = subprocess.run([program, str(kind)], capture_output=True, text=True, check=True).stdout.split()
    bad, used = int(out[0]), int(out[1])
    assert bad == 0
    assert kind in (-1, 6, 7) or used > 0.8 * 1024 * 256 * 64
