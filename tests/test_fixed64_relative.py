"""The parts of the bond-order angle terms that run over many sizes
(csrc/md_fixed64.cuh: the cutoff function and the sums, a fixed-point number and a
power of two each) against the host's extended precision, relative to their own
size.  Bars in units of 2^-53.  The exponential e^-a = v 2^-n, v above 0.49: four
units of 2^-56 (test_fixed64.py), so one; the cutoff multiplies it by a reciprocal
above 0.49 (three units, 0.8) and rounds a product above 0.24 (half a unit, 0.3):
2.1.  4 - 4 fc is four times that reciprocal, or its product with v: 2.1 of the
number itself.  Sums of eight terms of one sign lose a unit each below the largest
term, above 0.1: eight eighths of ten."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "moleculardynamics_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "md_fixed64.cuh"
using namespace mdgb;
typedef long double LD;
int main() {
  std::mt19937_64 gen(2);
  std::uniform_real_distribution<double> U(0, 1);
  const LD Q = std::ldexp((LD)1, 56), unit = std::ldexp((LD)1, -53);
  LD worst[3] = {0, 0, 0};
  auto see = [&](int k, LD got, LD ref) {
    worst[k] = std::fmax(worst[k], std::fabs(got - ref) / std::fabs(ref) / unit);
  };
  for (long i = 0; i < 1000000; i++) {
    const q56 r = toq(0.5 + 15.4 * (i < 1000 ? i / 1000.0 : U(gen)));
    q56 f, h;
    int n;
    cutoffq(r, f, n, h);
    const LD x = 4 * ((LD)r / Q - (LD)1.3f);
    see(0, std::ldexp((LD)f / Q, -n), 1 / (1 + std::exp(x)));
    see(1, (LD)h / Q, 4 / (1 + std::exp(-x)));
    SumQ s;
    LD ref = 0, refy = 0;
    for (int k = 0; k < 8; k++) {
      const q56 a = toq(0.1 + U(gen)), b = toq(0.1 + 7 * U(gen));
      const int e = (int)(U(gen) * 90);
      addq(s, a, -b, e);
      ref += std::ldexp((LD)a / Q, -e);
      refy -= std::ldexp((LD)b / Q, -e);
    }
    see(2, std::ldexp((LD)s.x / Q, -s.n), ref);
    see(2, std::ldexp((LD)s.y / Q, -s.n), refy);
  }
  for (LD w : worst) printf("%.3Lf ", w);
}
"""


def test_relative_errors(tmp_path):
    src = tmp_path / "relative.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "relative"
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no compiler")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    bars = [2.1, 2.1, 10.0]
    assert all(float(w) <= b for w, b in zip(out.split(), bars)), out
