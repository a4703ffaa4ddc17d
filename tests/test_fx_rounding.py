"""The rounding shift of the cluster transforms (csrc/nlm_kernels.h, fx_align), on the CPU."""
import os
import shutil
import subprocess

import pytest

from multimodenonlinearoptics_gb300 import build_ext

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "nlm_kernels.h"
int main() {
  for (int r = 0; r <= 8; r++) {   // every residue of v modulo 2^(r + 1), both signs
    long long sum = 0, far = 0;
    for (long long v = -4096; v < 4096; v++) {
      const long long q = nlm::fx_align(v, r);
      sum += (q << r) - v;
      far += q != std::llrint(std::ldexp((double)v, -r));   // nearest, ties to even
    }
    std::printf("%d %lld %lld\n", r, sum, far);
  }
  const long long big = (1LL << 60) - 1;
  std::printf("%lld %lld %lld\n", nlm::fx_align(big, 62), nlm::fx_align(-big, 61), nlm::fx_align(big, 40));
}
"""


def test_alignment_rounds_without_a_mean(tmp_path):
    """The error over all residues sums to zero for every shift, and no value is rounded but to nearest, ties to even."""
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    src, exe = tmp_path / "align.cpp", tmp_path / "align"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(build_ext._cuda_home(), "include"),
                    "-I" + build_ext.CSRC, "-I" + build_ext.INCLUDE, str(src), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for r in range(9):
        assert lines[r].split() == [str(r), "0", "0"]
    assert lines[9].split() == ["0", "0", str(1 << 20)]
