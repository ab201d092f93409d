"""Which small systems run all CG iterations in one kernel, and on how many CTAs,
when the device cannot place a cluster of 16 CTAs, or any cluster: 8 CTAs, or the
chain of kernels, and never a refused launch.  The rule is plain C++, compiled
here by itself."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include <cstdio>
#include <cstdlib>
#include "%s/ufc-fem-kernel_b200/csrc/resident_rule.h"
int main(int, char** v) {
  const int most = std::atoi(v[1]);
  for (int64_t s = 1; s <= 50; ++s)
    std::printf("%%d ", ufc::resident_ctas(s, [most](int g) { return g <= most; }));
  return 0;
}
"""


@pytest.mark.parametrize("most", [16, 15, 8, 7, 0])
def test_cta_count(tmp_path, most):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(SRC % ROOT)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-o", str(exe), str(src)], check=True)
    got = list(map(int, subprocess.run([str(exe), str(most)], check=True, capture_output=True, text=True).stdout.split()))
    for slices, g in zip(range(1, 51), got):
        if slices <= 4:
            want = 1
        elif slices > 48:
            want = 0
        else:
            want = next((k for k in (min(slices, 16), min(slices, 8)) if k <= most), 0)
        assert g == want, (slices, g)
        assert g == 0 or -(-slices // g) <= 16  # slices of a CTA: at most one warp each
