"""The quotients formed without an FP64 division (fortrancfd_gb300/csrc/idiv.h:
rcp_int / div_int, div_3, const_div / div_const) and the integer products
and root (mul_int, mul_k, sqrt_int), compiled as plain C++ and compared bit for bit with the
host's IEEE operations: random operands over the
whole exponent range, quotients next to a rounding midpoint (random and solved
for), zeros, subnormals, infinities and NaN, with the float seed of the
reciprocal displaced by its error bound either way."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fortrancfd_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <random>
#include "idiv.h"
using namespace gbmg;
static std::mt19937_64 g(1);
static long bad = 0, n = 0;
static int modes[4];
static double any(int lo, int hi) {
  uint64_t m = g() & 0xfffffffffffffull;
  switch (g() % 8) {
    case 0: m &= ~0ull << (g() % 52); break;
    case 1: m |= (1ull << (g() % 52)) - 1; break;
    case 2: m = 0xfffffffffffffull >> (g() % 52); break;
    case 3: m = g() % 4; break;
    case 4: m = 0xfffffffffffffull - (g() % 4); break;
    default: break;
  }
  return idiv_double((uint64_t)(lo + g() % (hi - lo + 1)) << 52 | m | ((g() & 1) << 63));
}
static void same(double x, double y, double a, double b, const char* what) {
  ++n;
  if (idiv_bits(x) != idiv_bits(y) && !(x != x && y != y) && bad++ < 10)
    std::printf("%s: %a / %a gives %a, not %a\n", what, a, b, x, y);
}
static const double edge[] = {0.0, -0.0, 4.9e-324, -2.3e-308, 1.0, -1.0, 3.0, INFINITY, -INFINITY,
                              NAN, 1.7976931348623157e308, 2.2250738585072014e-308};
int main() {
  for (int sh = -1; sh <= 1; ++sh) {
    idiv_seed_shift() = sh;
    for (long i = 0; i < 1000000; ++i) {
      const bool wide = i % 4 == 0;
      const double b = wide ? any(0, 2047) : any(900, 1100);
      const double a = i % 4 == 3 ? std::fabs(b) * any(1000, 1046) : wide ? any(0, 2047) : any(900, 1100);
      same(div_int(a, rcp_int(b)), a / b, a, b, "div_int");
      same(div_int(a, rcp_int(std::fabs(b))), a / std::fabs(b), a, std::fabs(b), "div_int");
      for (int s = 0; s < 3; ++s) same(div_3(a, s), a / (3 << s), a, 3 << s, "div_3");
      same(mul_int(a, b), a * b, a, b, "mul_int");
      same(mul_int(a, a), a * a, a, a, "mul_int");
      // short significands: products that end in a tie
      const double c = idiv_double(idiv_bits(a) & (~0ull << (20 + g() % 12)));
      const double d = idiv_double(idiv_bits(b) & (~0ull << (20 + g() % 12)));
      same(mul_int(c, d), c * d, c, d, "mul_int tie");
      same(mul_k<3>(a), 3.0 * a, a, 3, "mul_k");
      same(mul_k<5>(a), 5.0 * a, a, 5, "mul_k");
      same(mul_k<7>(a), 7.0 * a, a, 7, "mul_k");
      same(mul_k<11>(a), 11.0 * a, a, 11, "mul_k");
      same(mul_k<13>(a), 13.0 * a, a, 13, "mul_k");
      same(mul_k<15>(a), 15.0 * a, a, 15, "mul_k");
      same(sqrt_int(std::fabs(a)), std::sqrt(std::fabs(a)), a, 0, "sqrt_int");
      // squares of 53-bit values and their neighbours: roots next to a double
      const double q = idiv_double((idiv_bits(a) & 0xfffffffffffffull) | (1023ull + i % 2) << 52);
      for (int d = -2; d <= 2; ++d) {
        const double sq = idiv_double(idiv_bits(q * q) + (uint64_t)(int64_t)d);
        same(sqrt_int(sq), std::sqrt(sq), sq, 0, "sqrt_int square");
      }
      same(scale2<-1>(a), 0.5 * a, a, 0.5, "scale2");
      same(scale2<-2>(a), 0.25 * a, a, 0.25, "scale2");
      same(scale2<1>(a), 2.0 * a, a, 2, "scale2");
    }
    for (double a : edge) {
      for (double b : edge) same(mul_int(a, b), a * b, a, b, "mul_int edge");
      same(mul_k<3>(a), 3.0 * a, a, 3, "mul_k edge");
      same(sqrt_int(a), std::sqrt(a), a, 0, "sqrt_int edge");
      same(mul_k<13>(a), 13.0 * a, a, 13, "mul_k edge");
      same(scale2<-1>(a), 0.5 * a, a, 0.5, "scale2 edge");
      same(scale2<-2>(a), 0.25 * a, a, 0.25, "scale2 edge");
      same(scale2<1>(a), 2.0 * a, a, 2, "scale2 edge");
    }
    for (double a : edge)
      for (double b : edge) same(div_int(a, rcp_int(b)), a / b, a, b, "div_int edge");
    // a 2^s = b (2k+1) + d with a small d: the quotients nearest to a midpoint
    for (long i = 0; i < 100000; ++i) {
      const uint64_t B = (g() & 0xfffffffffffffull) | (1ull << 52) | 1;
      uint64_t inv = 1;
      for (int j = 0; j < 6; ++j) inv *= 2 - B * inv;
      for (int d = -3; d <= 3; d += 2)
        for (int s = 53; s <= 54; ++s) {
          const uint64_t M = ((uint64_t)(int64_t)(-d) * inv) & ((1ull << s) - 1);
          const uint64_t A = (uint64_t)(((unsigned __int128)B * M + d) >> s);
          if (A < (1ull << 52) || A >= (1ull << 53)) continue;
          same(div_int((double)A, rcp_int((double)B)), (double)A / (double)B, (double)A, (double)B,
               "div_int midpoint");
        }
    }
  }
  for (double a : edge)
    for (int s = 0; s < 3; ++s) same(div_3(a, s), a / (3 << s), a, 3 << s, "div_3 edge");
  // constant divisors: spacings, their squares, whole numbers, random
  for (int k = 0; k < 3000; ++k) {
    double h;
    switch (k % 6) {
      case 0: h = 1.0 / (2 + g() % 2000); break;
      case 1: h = 1.0 / (2 + g() % 1000); h *= h; break;
      case 2: h = (double)(1 + g() % 3000); break;
      case 3: h = std::ldexp((double)(g() >> 11), -60 + (int)(g() % 20)); break;
      case 4: h = -0.01 * (1 + g() % 500); break;
      default: h = std::ldexp(1.0 + (g() % 7) / 8.0, (int)(g() % 140) - 70);
    }
    const ConstDiv c = const_div(h);
    modes[c.mode]++;
    for (double a : edge) {
      same(div_const(c, a), a / h, a, h, "div_const edge");
      same(div_const_i(const_div_i(h), a), a / h, a, h, "div_const_i edge");
    }
    for (int i = 0; i < 600; ++i) {
      double x = any(700, 1300);
      if (i % 3 == 0) {
        const double m = std::ldexp((double)((g() >> 11) | (1ull << 52)), -20);
        x = h * (m + 0.5 * std::ldexp(1.0, std::ilogb(m) - 52));
      }
      if (i % 7 == 0) x = any(0, 2047);
      same(div_const(c, x), x / h, x, h, "div_const");
      same(div_const_i(c, x), x / h, x, h, "div_const_i");
    }
  }
  std::printf("%ld %ld %d %d %d %d\n", n, bad, modes[0], modes[1], modes[2], modes[3]);
  return bad != 0;
}
"""


def test_quotients_are_the_ieee_quotients(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "drv.cpp", tmp_path / "drv"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    counts = [int(x) for x in r.stdout.split()]
    assert counts[0] > 10 ** 7 and counts[1] == 0
    assert all(m > 0 for m in counts[2:])  # every rule of const_div was met
