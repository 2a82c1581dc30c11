"""The integer forms of FP64 products, quotients and square roots
(csrc/md_exact64.cuh) against the host's IEEE arithmetic, bit for bit: random
mantissas, mantissas at the ends of the binade and with few bits set, seeds at
their exact value and one and two units off (the approximation instructions
they come from are within one and 2^-22.9)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "moleculardynamics_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "md_exact64.cuh"
using namespace mdgb;
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static double dbl(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static uint32_t fbits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static float flt(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
int main() {
  std::mt19937_64 gen(7);
  long bad[4] = {0, 0, 0, 0};
  for (long k = 0; k < 4000000; k++) {
    auto draw = [&](int kind) {
      const uint64_t u = gen();
      uint64_t m = u & kMant52;
      if (kind == 1) m = u % 16;
      if (kind == 2) m = kMant52 - (u % 16);
      if (kind == 3) m = (u % 4096) << 40;
      if (kind == 4) m = (((u % 4096) << 40) - (u >> 60)) & kMant52;
      return ((1023 - 60 + (u >> 53) % 120) << 52) | m;
    };
    const uint64_t a = draw((int)(k % 6)), b = draw((int)(k / 6 % 6));
    const int off = (int)(k % 5) - 2;  // units of the seed
    bad[0] += imul64(a, b) != bits(dbl(a) * dbl(b));
    uint32_t f = 0x3F800000u | (uint32_t)((b >> 29) & 0x7FFFFF);
    uint32_t y = fbits((float)(1.0 / (double)flt(f))) + off;
    bad[1] += ircp64_seeded(b, seed_fraction(y)) != bits(1.0 / dbl(b));
    f = ((b >> 52) & 1 ? 0x3F800000u : 0x40000000u) | (uint32_t)((b >> 29) & 0x7FFFFF);
    y = fbits((float)(1.0 / std::sqrt((double)flt(f)))) + off;
    uint64_t sq;
    const double root = std::sqrt(dbl(b));
    bad[2] += isqrt64_seeded(b, seed_fraction(y), sq) != bits(root) || sq != bits(root * root);
    bad[3] += idiv64_const(a, b, divisor_fraction(b)) != bits(dbl(a) / dbl(b));
  }
  printf("%ld %ld %ld %ld\n", bad[0], bad[1], bad[2], bad[3]);
}
"""


def test_integer_arithmetic_is_correctly_rounded(tmp_path):
    src = tmp_path / "exact64.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "exact64"
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I", CSRC,
                        str(src), "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no compiler")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out.split() == ["0", "0", "0", "0"]
