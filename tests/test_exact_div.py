"""Quotients by a shared reciprocal (csrc/exact_div.cuh) are the bits of the
IEEE division.  The header is compiled for the host, where the seed is cut to
19 bits (worse than the device's), and compared with '/' on random operands,
divisors with extreme significands, quotients near the middle of two floats,
and the operands that take the division itself.  tests/test_gpu_exact_div.py
does the same with the device's seed."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "harm_finalwham_b200", "csrc")

SOURCE = r"""
#include "exact_div.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace hg;
static double make(uint64_t m, int e, bool neg) {
  uint64_t u = ((uint64_t)(1023 + e) << 52) | (m & ((1ull << 52) - 1)) | ((uint64_t)neg << 63);
  double x;
  memcpy(&x, &u, 8);
  return x;
}
static bool bits(double x, double y) { return memcmp(&x, &y, 8) == 0 || (x != x && y != y); }
int main(int argc, char **argv) {
  const int kind = atoi(argv[1]);
  std::mt19937_64 r(17 + kind);
  long bad = 0, used = 0;
  for (long n = 0; n < 4000000; n++) {
    uint64_t ma = r(), mb = r();
    int ea = (int)(r() % 60) - 30, eb = (int)(r() % 60) - 30;
    if (kind == 1) mb = ~(r() % 64);                        // significand near two
    if (kind == 2) mb = r() % 64;                           // near one
    if (kind == 3) { ma = ~(r() % 64); mb = ~(r() % 1024); }
    double b = make(mb, eb, false), a = make(ma, ea, r() & 1);
    if (kind == 4) {                                        // quotient near a middle
      const long double mid = (long double)make(r(), 0, false) + 0x1p-53L;
      a = (double)(mid * (long double)b);
    }
    if (kind == 5) { a = make(ma, (int)(r() % 1400) - 700, r() & 1); b = make(mb, (int)(r() % 400) - 200, false); }
    const Divisor<double> d = make_divisor(b);
    if (d.ok) { used++; if (!bits(d.y, 1.0 / b)) bad++; }
    double num[3] = {a, -a, a}, q[3];
    if (kind == 6) {                                        // what takes the division
      const double odd[] = {0.0, -0.0, 4e-324, -1e-310, 1e-250, 1e300, INFINITY, -INFINITY, NAN, 1.0};
      num[1] = odd[n % 10];
      num[2] = odd[(n / 10) % 10];
      const double den[] = {b, 1e-100, 1e100, 5e-324, INFINITY, NAN, make(~0ull, eb, false), 0.0};
      b = den[(n / 100) % 8];
    }
    if (kind == 7) {                                        // negative divisors, zero numerators among the others
      b = -b;
      if (n % 3 == 0) num[n % 2] = n % 4 < 2 ? 0.0 : -0.0;
    }
    div_n<3>(num, kind >= 6 ? known_divisor(b, kept_rcp(b)) : d, q);
    for (int i = 0; i < 3; i++) if (!bits(q[i], num[i] / b)) bad++;
  }
  printf("%ld %ld\n", bad, used);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_div")
    (d / "t.cc").write_text(SOURCE)
    exe = str(d / "t")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", CSRC, "-o", exe, str(d / "t.cc")], check=True)
    return exe


@pytest.mark.parametrize("kind", range(8))
def test_quotients_are_the_divisions_bits(program, kind):
    out = subprocess.run([program, str(kind)], capture_output=True, text=True, check=True).stdout.split()
    bad, used = int(out[0]), int(out[1])
    assert bad == 0
    assert kind >= 6 or used > 3_000_000
