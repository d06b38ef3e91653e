"""Which classes the autotuner chooses a kernel variant for: those whose kernels differ by
variant (the launch_jk cases), not those that run one kernel in all of them."""

import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tonto_b200", "csrc")

PROGRAM = r"""
#include "tf_host.h"
#include <cstdio>
int main() {
  for (int a = 0; a < 4; ++a) for (int b = 0; b <= a; ++b)
    for (int c = 0; c <= a; ++c) for (int d = 0; d <= c; ++d)
      if ((c < a || d <= b) && tf::has_variants(a, b, c, d)) std::printf("%d%d%d%d\n", a, b, c, d);
}
"""


def test_classes_with_variants(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "p")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", exe, str(tmp_path / "p.cpp")], check=True)
    got = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    want = []
    for f in sorted(os.listdir(CSRC)):
        if f.startswith("tf_jk_"):
            want += ["".join(m) for m in re.findall(r"TF_JK_CASE\(launch_jk, (\d), (\d), (\d), (\d)\)",
                                                    open(os.path.join(CSRC, f)).read())]
    assert sorted(got) == sorted(want) and len(want) == 12


def test_the_autotuner_asks():
    code = open(os.path.join(CSRC, "tontofock.cu")).read()
    tune = code[code.index("int tf_autotune("):code.index("int tf_set_shard(")]
    assert "if (has_variants(" in tune
