"""The fixed-point arithmetic of the bond-order angle terms
(csrc/md_fixed64.cuh, 56 bits after the point) against the host's extended
precision.  Bars in units of 2^-56, from the error terms: a conversion or a
product cuts off less than one; a reciprocal or root adds the truncations of two
scaled corrections to a cubic remainder below one (3); the exponential adds those
of three products, its cut series and the rounded table (4); back in FP64 half a
unit of 2^-53 relative, with the tie rounded up (0.5)."""
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
#include "md_fixed64.cuh"
using namespace mdgb;
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
static uint32_t fbits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static float flt(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
typedef long double LD;
int main() {
  std::mt19937_64 gen(1);
  std::uniform_real_distribution<double> U(0, 1);
  const LD Q = std::ldexp((LD)1, 56);
  LD worst[7] = {0, 0, 0, 0, 0, 0, 0};
  auto see = [&](int k, LD e) { worst[k] = std::fmax(worst[k], std::fabs(e)); };
  for (long i = 0; i < 2000000; i++) {
    const int off = (int)(i % 3) - 1;  // units of the seed
    const double a = (U(gen) * 2 - 1) * 7.9, b = (U(gen) * 2 - 1) * 7.9;
    const q56 qa = toq(a), qb = toq(b);
    see(0, (LD)qa - (LD)a * Q);
    see(1, (LD)mulq(qa, qb) - (LD)qa * (LD)qb / Q);
    see(2, ((LD)fromq(qa) * Q - (LD)qa) / (std::fabs((LD)a) * Q) * std::ldexp((LD)1, 53));
    q56 den = kQOne + (q56)(U(gen) * (double)kQOne);
    if (i % 97 == 0) den = kQOne;
    if (i % 101 == 0) den = 2 * kQOne;
    uint32_t f = 0x3F800000u + (uint32_t)((uint64_t)(den - kQOne) >> 33);
    uint32_t y = seed_fraction(fbits((float)(1.0 / (double)flt(f))) + off);
    see(3, (LD)rcpq_seeded(den, y) - Q * Q / (LD)den);
    const double r2 = std::exp2(U(gen) * 9.99 - 2);
    f = ((bits(r2) >> 52) & 1 ? 0x3F800000u : 0x40000000u) | (uint32_t)((bits(r2) >> 29) & 0x7FFFFF);
    y = seed_fraction(fbits((float)(1.0 / std::sqrt((double)flt(f)))) + off);
    q56 r, ir;
    rsqrtq_seeded(bits(r2), y, r, ir);
    see(4, ((LD)r - std::sqrt((LD)r2) * Q) / std::fmax((LD)1, std::sqrt((LD)r2)));
    see(5, (LD)ir - Q / std::sqrt((LD)r2));
    const q56 x = i % 89 ? toq(U(gen) * 40) : 0;
    see(6, (LD)expnegq(x) - std::exp(-(LD)x / Q) * Q);
  }
  for (LD w : worst) printf("%.3Lf ", w);
}
"""


def test_fixed_point_errors(tmp_path):
    src = tmp_path / "fixed64.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "fixed64"
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no compiler")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    bars = [1.0, 1.0, 0.501, 3.0, 3.0, 3.0, 4.0]
    assert all(float(w) <= b for w, b in zip(out.split(), bars)), out
