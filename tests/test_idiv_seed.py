"""The float seeds of the integer quotient and root (idiv.h) over the whole error bound
that their exactness rests on.  CPU: the seed displaced by up to two ulps of the
rounded value wherever that stays within the bound, against the host's division and
root.  GPU: the error of the instructions that give the seeds, over every float that
they are given."""
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
static std::mt19937_64 g(7);
static long bad = 0, n = 0, two = 0;
static void same(double x, double y, double a, double b) {
  ++n;
  if (idiv_bits(x) != idiv_bits(y) && bad++ < 10) std::printf("%a, %a: %a, not %a\n", a, b, x, y);
}
// the float whose reciprocal (root) rcp_int (sqrt_int) asks for
static float lead(double b) {
  return idiv_float(0x3f800000u | (uint32_t)(idiv_bits(b) >> 29 & 0x7fffffu));
}
static float lead_root(double a) {
  const uint64_t u = idiv_bits(a);
  return idiv_float((u >> 52 & 1 ? 0x3f800000u : 0x40000000u) | (uint32_t)(u >> 29 & 0x7fffffu));
}
static double any() {
  uint64_t m = g() & 0xfffffffffffffull;
  switch (g() % 6) {
    case 0: m &= ~0ull << (g() % 52); break;
    case 1: m |= (1ull << (g() % 52)) - 1; break;
    case 2: m = 0xfffffffffffffull >> (g() % 52); break;
    case 3: m = 0xfffffffffffffull - (g() % 4); break;
    default: break;
  }
  return idiv_double((1000 + g() % 46) << 52 | m);
}
int main() {
  const double rcp_bound = 0x1p-23, root_bound = std::exp2(-22.9);
  for (int sh = -2; sh <= 2; ++sh) {
    idiv_seed_shift() = sh;
    for (long i = 0; i < 2000000; ++i) {
      const double a = any(), b = any();
      const double x = lead(b), r = lead_root(a);
      if (std::fabs((double)idiv_seed((float)x) * x - 1.0) <= rcp_bound) {
        two += sh == 2 || sh == -2;
        same(div_int(a, rcp_int(b)), a / b, a, b);
      }
      if (std::fabs((double)isqrt_seed((float)r) * std::sqrt(r) - 1.0) <= root_bound) {
        same(sqrt_int(a), std::sqrt(a), a, 0);
        const double q = idiv_double((idiv_bits(a) & 0xfffffffffffffull) | 1023ull << 52);
        for (int d = -1; d <= 1; ++d) {
          const double s = idiv_double(idiv_bits(q * q) + (uint64_t)(int64_t)d), l = lead_root(s);
          if (std::fabs((double)isqrt_seed((float)l) * std::sqrt(l) - 1.0) <= root_bound)
            same(sqrt_int(s), std::sqrt(s), s, 0);
        }
      }
    }
  }
  std::printf("%ld %ld %ld\n", n, bad, two);
  return bad != 0;
}
"""

SEEDS = r"""
#include <cstdio>
#include "idiv.h"
using namespace gbmg;
// largest error (relative, in units of 2^-40) of the seeds over every float
__global__ void seeds(unsigned long long* worst) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 1u << 24) return;
  if (i < 1u << 23) {
    const float x = __uint_as_float(0x3f800000u + i);
    const double e = fabs((double)idiv_seed(x) * x - 1.0);
    atomicMax(worst, (unsigned long long)(e * 0x1p40));
  }
  const float x = __uint_as_float(0x3f800000u + i);
  const double e = fabs((double)isqrt_seed(x) * sqrt((double)x) - 1.0);
  atomicMax(worst + 1, (unsigned long long)(e * 0x1p40));
}
int main() {
  unsigned long long* d = nullptr;
  unsigned long long h[2] = {0, 0};
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 2;
  seeds<<<(1 << 24) / 256, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu %llu\n", h[0], h[1]);
  cudaFree(d);
  return 0;
}
"""


def test_exact_over_the_bound(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "drv.cpp", tmp_path / "drv"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    n, bad, two = (int(v) for v in r.stdout.split())
    assert n > 10 ** 7 and bad == 0
    assert two > 10 ** 5  # displacements of two ulps within the bound


@pytest.mark.gpu
def test_seed_errors(cuda, tmp_path):
    from fortrancfd_gb300 import build
    src, exe = tmp_path / "seeds.cu", tmp_path / "seeds"
    src.write_text(SEEDS)
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-I", CSRC, str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, check=True)
    rcp, root = (int(v) * 2.0 ** -40 for v in r.stdout.split())
    assert 0 < rcp <= 2.0 ** -23
    assert 0 < root <= 2.0 ** -22.9
