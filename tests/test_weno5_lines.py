"""The FP64 WENO5 pieces that weno5_kernel calls (indicator class from signs
and exponents, shared reciprocals, quotients left unformed where a product
decides) give the bits of the plain routines, over lines of every kind: flat
and rough ones, any magnitude, squares that overflow, denormals, infinities
and NaN.  Both run on the host, along lines as the kernel marches them."""
import subprocess

import pytest

from tests import host_device

SOURCE = r"""
#include "weno5.cuh"
using namespace hg;
constexpr int N = 16;  // output cells; cell c at y[c + 5]
static bool same(double a, double b) { return a == b || (a != a && b != b); }
static void plain(const double *y, const double *S, double *L, double *R) {
  double m0[N + 6], w[N + 6][3], lof[N + 2];
  bool cu[N + 6];
  for (int s = 0; s < N + 6; s++) {
    const double *u = y + s + 2;
    cu[s] = w5::cusp(u, u);
    m0[s] = cu[s] ? 0.0 : w5::mono(u, u);
    w5::unopt3(m0[s], u, u, w[s]);
  }
  for (int s = 0; s < N + 2; s++) lof[s] = w5::ratio_lof(w[s + 2], w[s][0], w[s + 4][2], cu[s + 2] ? 1.0 : 0.0);
  for (int s = 0; s < N; s++) {
    const double f = w5::wmax(w5::wmax(lof[s + 1], S[s] * lof[s + 2]), S[s] * lof[s]);
    w5::faces(y + s + 5, y + s + 5, m0[s + 3], cu[s + 3], w[s + 3], f, L + s, R + s);
  }
}
static void marched(const double *y, const double *S, double *L, double *R) {
  int code[N + 6];
  double w[N + 6][3], lof[N + 2];
  for (int s = 0; s < N + 6; s++) {
    const double *u = y + s + 2;
    code[s] = w5::code_of<double>(u, u);
    w5::weights3<double>(code[s], u, u, w[s]);
  }
  for (int s = 0; s < N + 2; s++)
    lof[s] = w5::lower_fraction<double>(code[s + 2], w[s + 2][0], w[s + 2][2], w[s][0], w[s + 4][2]);
  for (int s = 0; s < N; s++) {
    const double f = w5::wmax(w5::wmax(lof[s + 1], S[s] * lof[s + 2]), S[s] * lof[s]);
    w5::face_values<double>(code[s + 3], y + s + 5, y + s + 5, w[s + 3], f, L + s, R + s);
  }
}
int main(int argc, char **argv) {
  const int kind = atoi(argv[1]);
  std::mt19937_64 r(31 + kind);
  std::uniform_real_distribution<double> U(-1, 1);
  std::normal_distribution<double> G;
  double y[N + 10], S[N], a[2][N], b[2][N];
  long bad = 0;
  for (long t = 0; t < 100000; t++) {
    const double base = r() % 3 ? 1.0 : 0.0, amp = pow(10., -16 + 8 * (U(r) + 1));
    const double scale = pow(10., 307 * U(r)), phase = 3 * U(r);
    for (int i = 0; i < N + 10; i++) {
      const double rough = base + amp * G(r), wave = sin(0.1 * i + phase) + base;
      if (kind == 0) y[i] = rough;
      if (kind == 1) y[i] = wave * scale;                                  // smooth, at any scale
      if (kind == 2) y[i] = wave * scale * (1 + 1e-3 * amp * G(r));
      if (kind == 3) y[i] = pow(10., 308 * U(r));                          // any magnitude, cell by cell
      if (kind == 4) y[i] = pow(10., 150 + 10 * U(r)) * (r() % 2 ? 1 : -1);  // squares overflow or not
      if (kind == 5) y[i] = wave * pow(10., -300 - 8 * base) * (1 + amp * G(r));
      if (kind == 6) y[i] = r() % 4 ? 1.0 : 1.0 + amp * (double)(r() % 3);
      if (kind == 7) y[i] = rough;
    }
    if (kind == 7)
      for (int q = 1 + r() % 3; q > 0; q--) {
        const double odd[] = {INFINITY, -INFINITY, NAN, -NAN, 1.7e308, -1.7e308, 1e200, 0.0, -0.0, 5e-324};
        y[r() % (N + 10)] = odd[r() % 10];
      }
    for (int i = 0; i < N; i++) S[i] = kind == 7 && r() % 20 == 0 ? NAN : (r() % 3 ? U(r) : (double)(r() % 2));
    plain(y, S, a[0], a[1]);
    marched(y, S, b[0], b[1]);
    for (int i = 0; i < 2 * N; i++) bad += !same(a[i / N][i % N], b[i / N][i % N]);
  }
  printf("%ld\n", bad);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return host_device.build(tmp_path_factory.mktemp("weno5_lines"), SOURCE)


@pytest.mark.parametrize("kind", range(8))
def test_marched_lines_have_the_plain_routines_bits(program, kind):
    out = subprocess.run([program, str(kind)], capture_output=True, text=True, check=True).stdout
    assert int(out) == 0
