"""``csrc/dqb_scalar.cuh`` compiled by the host compiler (the same IEEE operations, FMA
included): the quotient is the division's to the last bit, the fifth root within an ulp."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
using std::fma;
static float __frcp_rn(float x) { return 1.0f / x; }
#include "dqb_scalar.cuh"

static bool same(double a, double b) { return std::memcmp(&a, &b, 8) == 0 || (a != a && b != b); }

int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> u(-99.0, 99.0), wide(-290.0, 290.0);
  long quotients = 0;
  double root = 0;
  for (int i = 0; i < 2000000; ++i) {
    const double y = std::exp2(u(g)), x = std::exp2(2 * u(g));
    quotients += !same(dqb::ratio(x, y), x / y) + !same(dqb::ratio(0.0, y), 0.0);
    const double yw = std::exp2(wide(g)), xw = std::exp2(wide(g));  // either side of the ranges
    quotients += !same(dqb::ratio(xw, yw), xw / yw);
  }
  const double inf = INFINITY, nan = NAN, edge[] = {0.0, 5e-324, 1e-300, 1e-31, 1e-30, 1.0, 1e30, 1e31, 1e271, 1e308, inf, nan};
  for (double y : edge)
    for (double x : {0.0, 1.0, 1e269, 1e271, 1e308, inf, nan}) quotients += !same(dqb::ratio(x, y), x / y);
  for (int i = 0; i < 200000; ++i) {
    const double e = std::exp2(u(g));
    int k;
    const long double t = std::pow((long double)e, -0.2L);
    std::frexp((double)t, &k);
    root = std::fmax(root, (double)(std::fabs((long double)dqb::inverse_fifth_root(e) - t) / std::ldexp(1.0L, k - 53)));
  }
  for (double e : edge) quotients += !(e > 1e-30 && e < 1e30) && !same(dqb::inverse_fifth_root(e), std::pow(e, -0.2));
  std::printf("%ld %.3f\n", quotients, root);
}
"""


@pytest.fixture(scope='module')
def result(tmp_path_factory):
    d = tmp_path_factory.mktemp('scalar')
    (d / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-O2', '-std=c++17', '-ffp-contract=off', '-Wno-unknown-pragmas',
                    '-I', os.path.join(ROOT, 'dynamiqs_b200', 'csrc'), 'main.cpp', '-o', 'main'], cwd=d, check=True)
    out = subprocess.run([str(d / 'main')], check=True, capture_output=True, text=True).stdout.split()
    return int(out[0]), float(out[1])


def test_quotients_are_the_divisions(result):
    assert result[0] == 0


def test_fifth_root_within_an_ulp(result):
    assert result[1] <= 1.0  # the last Newton step: half an ulp of its sum, the rest of its addend
