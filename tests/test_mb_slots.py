"""Slots of the forces on third bodies (csrc/md_forces.h): 64 an atom, no more than
the short lists hold, no more than a quarter of the free memory, down to none."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "moleculardynamics_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "md_forces.h"
int main() {
  const unsigned long long G = 1ull << 30;
  const long long n[] = {172, 4096, 50000000, 50000000, 50000000, 67000000, 172};
  const int pitch[] = {4, 224, 224, 224, 224, 224, 224};
  const unsigned long long free_b[] = {G, 200 * G, 200 * G, 20 * G, 3 * G, 0, 1000};
  for (int k = 0; k < 7; k++) printf("%d ", mdgb::mb_slot_count(n[k], pitch[k], free_b[k]));
}
"""


def test_slot_count(tmp_path):
    src = tmp_path / "slots.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "slots"
    inc = os.path.join(os.path.dirname(os.path.dirname(CSRC)), "include")
    r = subprocess.run(["nvcc", "-std=c++17", "-I", CSRC, "-I", inc, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no compiler")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    # 3 doubles a slot: 50 million atoms take 1.2 GB for each
    assert [int(v) for v in out.split()] == [4, 64, 32, 4, 0, 0, 0]
