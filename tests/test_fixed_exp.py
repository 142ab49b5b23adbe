"""The exponential and the intervals' arguments of the general smoothness'
tables (csrc/sv_fix.cuh), compiled as host C++ against long double, octave by
octave: e^-c within 4 units of 2^-58 (its argument's rounding, the polynomial's
and three truncated products), its mean error within half a unit (a shift of
2^-58 common to all near pairs is what the fixed-point arithmetic may not
have), t within 2 units, fx_to_double to nearest, ties up."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyscaledvecchia_gb300", "csrc")

DRIVER = r"""
#include "sv_fix.cuh"
#include <cstdio>
#include <cmath>
using namespace sv;
typedef long double LD;
static uint64_t st = 88172645463325252ULL;
static uint64_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
int main() {
  const LD u = std::ldexp((LD)1, 58), r2 = std::sqrt((LD)2);
  for (int e = -30; e < 9; ++e) {
    LD mx = 0, sum = 0, tm = 0;
    long bad = 0;
    const int N = 40000;
    for (int it = 0; it < N; ++it) {
      const uint64_t f = it == 0 ? 0 : it == 1 ? (1ull << 52) - 1 : rnd() >> 12;
      const LD x = 1 + std::ldexp((LD)f, -52), c = std::ldexp(x, e);
      int n;
      const uint64_t v = fx_exp_neg(f, e, kFxExp2, n);
      const LD err = (std::ldexp((LD)v, -62 - n) - std::exp(-c)) * u;
      mx = std::fmax(mx, std::fabs(err));
      sum += err;
      const bool up = x >= r2;
      const LD lo = up ? r2 : 1, hi = up ? 2 : r2;
      tm = std::fmax(tm, std::fabs(std::ldexp((LD)fx_tab_t(f, up), -58) - (2 * x - lo - hi) / (hi - lo)) * u);
      const int z = __builtin_clzll(v);
      const uint64_t w = ((v << z) >> 11) + ((v << z) >> 10 & 1);
      bad += fx_to_double(v, -62 - n) != std::ldexp((double)w, 11 - z - 62 - n);
    }
    std::printf("%d %.4Lf %.4Lf %.4Lf %ld\n", e, mx, sum / N, tm, bad);
  }
}
"""


def test_octaves(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    subprocess.run([gxx, "-O2", "-std=gnu++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for row in out[:-1]:
        e, mx, mean, t, bad = (float(v) for v in row.split())
        assert mx <= 4 and abs(mean) <= 0.5 and t <= 2 and bad == 0, row
