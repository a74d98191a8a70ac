"""Rounding of the polynomial SU(3) projection: over sums of links near one SU(3)
matrix (spread eps, from fields smeared for long to rough ones) its error may be
no larger than that of the matrix steps, in both precisions. Host build of the
header (fused multiply-adds as on the device); the exact projection of the same
rounded sum comes from extended precision.

The matrix steps are those of the smearing kernels: FP64 with the early exit,
FP32 (from a sum scaled to mean square 1 for the 12-real links) until the defect
is 2e-5 and one FP64 step. Both are sums of a few independent roundings, so over
some 3000 matrices (50000 numbers) their rms is known to 0.5%.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "general_code_b200" / "csrc"

SOURCE = r"""
#include "gc_algebra.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace gc;
typedef long double ld;
template <class T, class S> static SU3<T> to(const SU3<S> &a) {
  SU3<T> b;
  for (int k = 0; k < 9; k++)
    b.e[k / 3][k % 3] = {T(a.e[k / 3][k % 3].re), T(a.e[k / 3][k % 3].im)};
  return b;
}
static SU3<ld> limit(SU3<ld> a) {
  for (int i = 0; i < 12; i++)
    a = ns_step(a);
  return a;
}
static std::mt19937_64 rng(3);
static SU3<ld> near_unit(double eps) {
  std::normal_distribution<double> n;
  SU3<ld> a;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      a.e[i][j] = {(i == j) + eps * n(rng), eps * n(rng)};
  return limit(a);
}
static double sq(const SU3<double> &a, const SU3<ld> &x, int rows) {
  double s = 0;
  for (int k = 0; k < 3 * rows; k++) {
    const ld re = a.e[k / 3][k % 3].re - x.e[k / 3][k % 3].re;
    const ld im = a.e[k / 3][k % 3].im - x.e[k / 3][k % 3].im;
    s += double(re * re + im * im);
  }
  return s;
}
int main(int, char **argv) {
  const double eps = std::atof(argv[1]);
  double e[6] = {0, 0, 0, 0, 0, 0};
  long n = 0;
  for (int it = 0; it < 5000; it++) {
    SU3<ld> H = near_unit(0.3), S;
    for (int i = 0; i < 4; i++)
      H = mul(H, near_unit(0.3));
    S = scale(mul(near_unit(eps), H), ld(0.5));
    for (int i = 0; i < 4; i++)
      S = add(S, scale(mul(near_unit(eps), H), ld(0.125)));
    const SU3<double> D = to<double>(S);
    const SU3<float> F = to<float>(S);
    SU3<double> P;
    SU3<float> Q;
    cx<float> z;
    // (H is no SU(3) matrix where 12 steps did not reach one)
    if (!polar_su3(D, P) || !polar_parts(F, Q, z))
      continue;
    n++;
    const SU3<ld> X = limit(to<ld>(D));
    e[0] += sq(P, X, 3);
    e[1] += sq(proj(D, 1e-14), X, 3);
    const SU3<ld> Y = limit(to<ld>(F));
    e[2] += sq(to<double>(polar_finish<false>(Q, z)), Y, 2);
    e[4] += sq(to<double>(polar_finish<true>(Q, z)), Y, 3);
    for (int norm = 0; norm < 2; norm++) {
      float f2 = 0;
      for (int k = 0; k < 9; k++)
        f2 += F.e[k / 3][k % 3].re * F.e[k / 3][k % 3].re +
              F.e[k / 3][k % 3].im * F.e[k / 3][k % 3].im;
      int m;
      const SU3<float> B = ns_until(norm ? scale(F, 1.f / sqrtf(f2 / 3.f)) : F, 2e-5f, 5, &m);
      const SU3<double> G = to<double>(to<float>(ns_step(to<double>(B))));
      e[norm ? 3 : 5] += sq(G, Y, norm ? 2 : 3);
    }
  }
  for (int i = 0; i < 6; i++)
    std::printf("%.6e ", e[i]);
  std::printf("%ld", n);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("rounding")
    (d / "rounding.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=fast", "-I",
                    str(CSRC), str(d / "rounding.cpp"), "-o", str(d / "rounding")], check=True)
    return str(d / "rounding")


@pytest.mark.parametrize("eps", [1e-6, 1e-4, 1e-3, 3e-3, 1e-2, 0.1, 0.2])
def test_no_further_off_than_the_matrix_steps(program, eps):
    *e, n = [float(v) for v in subprocess.run([program, str(eps)], capture_output=True, text=True,
                                              check=True).stdout.split()]
    assert n > 1500
    for polynomial, steps in zip(e[0::2], e[1::2]):
        assert polynomial <= steps
