"""The integer square root and division of the FP64 kernels (csrc/exact64.h)
against sqrt() and the division operator, compiled for the host: significands
next to powers of two, next to squares of rounding midpoints and quotients next
to midpoints, and the approximation off by twice the unit's error either way;
then the filament and ring velocities against the plain ones, with targets on
corners and lines, degenerate edges, infinities and extreme scales.  The bits
have to agree."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "volcanor_gb300" / "csrc"

PROGRAM = r"""
#include "exact64.h"
#include <random>
using namespace vlm;
using namespace vlm::exact64;
static bool same(double a, double b) { return bits(a) == bits(b) || (a != a && b != b); }
static bool same(d3 a, d3 b) { return same(a.x, b.x) && same(a.y, b.y) && same(a.z, b.z); }
int main() {
  std::mt19937_64 g(5);
  auto number = [&](int lo, int hi) {
    uint64_t man = g() & 0xfffffffffffffull;
    switch (g() % 6) {
      case 0: man &= 0xfff; break;
      case 1: man |= 0xffffffffff000ull; break;
      case 2: man = 0xfffffffffffffull - (man & 7); break;
      case 3: man &= 7; break;
    }
    return from_bits(((uint64_t)(lo + 1023 + (int)(g() % (uint64_t)(hi - lo))) << 52) | man);
  };
  for (int i = 0; i < 1000000; ++i) {
    double x = number(-400, 400);
    if (i % 3 == 0) {  // next to the square of a midpoint
      const uint64_t N = (1ull << 52) | (g() & 0xfffffffffffffull);
      unsigned __int128 t = (unsigned __int128)(2 * N + 1) * (2 * N + 1);
      int sh = 0;
      for (; t >> 53; t >>= 1) ++sh;
      x = ldexp((double)((uint64_t)t + g() % 3 - 1), sh - 106 + 2 * ((int)(g() % 100) - 50));
    }
    const Root r = root_of(x);
    const double s = value(r);
    if (!same(s, sqrt(x))) return 1;
    const uint64_t Z = reciprocal(r);
    double a[6] = {number(-800, 700), -number(-800, 700), s, nextafter(s, 0.0), nextafter(s, INFINITY), -0.0};
    a[0] = i & 1 ? a[0] : (double)((long double)s * ((long double)number(0, 1) + ldexpl(1, -53)));
    for (double d : a)
      if (!div_in_range(d) || !same(divide(d, r, Z), d / s)) return 2;
  }
  // any divisor: extremes of its significand, quotients next to midpoints, both signs
  for (int i = 0; i < 1000000; ++i) {
    const double d = (i & 1 ? -1.0 : 1.0) * number(-200, 200);
    const double a = i % 3 ? number(-800, 700) : (double)((long double)d * ((long double)number(0, 1) + ldexpl(1, -53)));
    if (!divisor_in_range(d) || !same(quotient(a, d), a / d) || !same(quotient(0.0, d), 0.0 / d)) return 5;
  }
  for (double d : {0.0, -0.0, 1e-310, 1e300, (double)INFINITY, (double)NAN, 3.0})
    for (double a : {0.0, 1.0, -2e-308, 1e308, (double)INFINITY, (double)NAN})
      if (!same(quotient(a, d), a / d)) return 6;
  std::uniform_real_distribution<double> U(-1, 1);
  for (int i = 0; i < 200000; ++i) {
    const double sc = i % 7 == 0 ? ldexp(1.0, (int)(g() % 1200) - 600) : 1.0;
    auto point = [&]() { return mk3(U(g) * sc, U(g) * sc, U(g) * sc); };
    d3 P = point(), c[4] = {point(), point(), point(), point()};
    const double rv[4] = {0.01 * sc, 0.0, 1e-3 * sc, 0.01 * sc};
    switch (g() % 10) {
      case 0: P = c[1]; break;
      case 1: P = 0.5 * (c[0] + c[1]); break;
      case 2: c[2] = c[1]; break;
      case 3: for (d3& q : c) q.z = P.z; break;
      case 4: P = c[0] + 1e-17 * c[1]; break;
      case 5: c[3].x = INFINITY; break;
      case 6: c[3].y = NAN; break;
    }
    if (!same(vr_vind64(P, c, rv), exact64::vr_vind(Unit{1.0, -0.0}, P, c, rv))) return 3;
    if (!same(exact64::unit(c[0]), unit3(c[0])) || !same(exact64::proj(P, c[1]), proj3(P, c[1])) ||
        !same(exact64::noproj(P, c[1]), noproj3(P, c[1])) || !same(exact64::norm(c[2]), norm3(c[2])))
      return 7;
    if (!same(fil_vind64(P, c[0], c[1], rv[0]), exact64::fil_vind(Unit{1.0, -0.0}, P, c[0], c[1], rv[0]))) return 4;
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("factor", ["1.0f", "(1.0f-5e-7f)", "(1.0f+5e-7f)"])
def test_integer_roots_and_quotients_are_correctly_rounded(tmp_path, factor):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}",
                           f"-DVLM_RSQRT32_FACTOR={factor}", str(src), "-o", str(exe)])
    assert subprocess.run([str(exe)]).returncode == 0
