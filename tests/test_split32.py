"""Coordinate differences of the surrogate's kernels (csrc/md_split32.cuh) against
extended precision: rounded once to FP32.  Bar: half a unit in the last place, a
thousandth of one for the second rounding, and the parts' own roundings, a dozen of
2^-48 of the coordinates (300 angstrom)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "moleculardynamics_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "md_split32.cuh"
using namespace mdgb;
typedef long double LD;
int main() {
  std::mt19937_64 gen(3);
  std::uniform_real_distribution<double> U(0, 1);
  double worst = 0;
  const LD parts = 12 * 300 * std::ldexp((LD)1, -48);
  for (long k = 0; k < 4000000; k++) {
    const double L = 20 + 280 * U(gen);
    const int img = (int)(k % 3) - 1;
    const double d = (U(gen) * 2 - 1) * 3 * std::pow(10.0, -3 * U(gen));
    // j near i, through a face where there is an image; often near the origin
    double xi = (U(gen) - 0.5) * (k % 5 ? L : 4.0);
    if (img) xi = img * (L / 2 - 2 * U(gen));
    const double xj = xi + d - img * L;
    const LD ref = (LD)xj + img * (LD)L - (LD)xi;
    const float got = diff32(split64(xj), split64(xi), img, split64(L));
    const float r = std::fabs((float)ref);
    const LD ulp = (LD)std::nextafterf(r, INFINITY) - r;
    const double off = (double)((std::fabs((LD)got - ref) - parts) / ulp);
    worst = off > worst ? off : worst;
  }
  printf("%.5f", worst);
}
"""


def test_difference_rounded_once(tmp_path):
    src = tmp_path / "split.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "split"
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no compiler")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert float(out) <= 0.501, out
