"""The three-operation division of the FP64 kernels (swm_div.cuh), compiled for
the host, against the machine's division: the same bits for every dividend,
divisors of every mantissa shape (ones, a single bit, random) in the range that
has a reciprocal, and everything outside it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = """
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline int __double2hiint(double x) { int64_t b; std::memcpy(&b, &x, 8); return int(b >> 32); }
inline int __double2loint(double x) { int64_t b; std::memcpy(&b, &x, 8); return int(b); }
"""

MAIN = """
#include "swm_div.cuh"
#include <cstdio>
#include <limits>
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double make(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static uint64_t mant(int kind) {
  const uint64_t all = (1ull << 52) - 1;
  switch (kind) {
    case 0: return rnd() & all;
    case 1: return all;
    case 2: return 0;
    case 3: return 1ull << (rnd() % 52);
    case 4: return all ^ (1ull << (rnd() % 52));
    case 5: return all >> (rnd() % 52);
    default: return rnd() & 15;
  }
}
static long bad = 0, n = 0;
static void check(double a, double b) {
  // kRecipLow, kRecipHigh
  const double rb = std::fabs(b) >= 0x1p-64 && std::fabs(b) <= 0x1p500
                        ? 1.0 / b : std::numeric_limits<double>::quiet_NaN();
  const double q = imodel::div_by(a, b, rb), e = a / b;
  ++n;
  if (bits(q) != bits(e) && !(q != q && e != e)) {
    if (bad++ < 5) std::printf("%a / %a: %a, not %a\\n", a, b, q, e);
  }
}
int main() {
  for (int k = 0; k < 400000; ++k) {
    const double m = make((1023ull << 52) | mant(int(rnd() % 7)));
    const double b = std::ldexp(m, int(rnd() % 580) - 72) * ((rnd() & 1) ? 1.0 : -1.0);
    // quotients close to a number or to the middle between two, and any others
    double a = make((1023ull << 52) | mant(int(rnd() % 7)));
    if (rnd() & 1) a = a * m;
    check(std::ldexp(a, int(rnd() % 2040) - 1000) * ((rnd() & 1) ? 1.0 : -1.0), b);
    check(a, 6.0);
    check(a, 6371220.0);
  }
  const double inf = std::numeric_limits<double>::infinity();
  const double sp[] = {0.0, -0.0, 1.0, -1.0, 3.0, 0x1p-1074, -0x1p-1074, 0x1p-1022, 0x1.fffffffffffffp1023,
                       0x1p-895, 0x1p896, 0x1p-64, 0x1.fffffffffffffp-64, 0x1.fffffffffffffp-65,
                       0x1p-959, 0x1p-960, 0x1p500, 0x1p501, 0x1p-501, 1e-12, inf, -inf, inf - inf};
  for (double a : sp)
    for (double b : sp) check(a, b);
  std::printf("%ld of %ld differ\\n", bad, n);
  return bad != 0;
}
"""


def test_division_by_a_known_divisor_is_division(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    (tmp_path / "cuda_runtime.h").write_text(SHIM)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "div")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(tmp_path), "-I",
                    os.path.join(ROOT, "imodel_gb300", "csrc"), "-x", "c++",
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
