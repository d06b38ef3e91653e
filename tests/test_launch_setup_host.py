"""A kernel's launch set-up (shared-memory attribute, resident blocks) holds for one device, so
it is made once per device, whatever threads ask first, and again after a failure.

tf_host.h holds no device code; this compiles its table for the host with a set-up that
counts."""

import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tonto_b200", "csrc")

PROGRAM = r"""
#include "tf_host.h"
#include <chrono>
#include <cstdio>
#include <thread>
struct Two { long long a, b; };
int main() {
  tf::PerDevice<Two> t;
  std::atomic<int> made[4] = {}, wrong{0};
  std::vector<std::thread> threads;
  for (int k = 0; k < 16; ++k)
    threads.emplace_back([&, k] {
      for (int i = 0; i < 200; ++i) {
        const int dev = (k + i) % 4;
        Two v{};
        const bool ok = t.get(dev, v, [&](Two& x) {
          x.a = 100 + dev;                       // half written while others ask
          std::this_thread::sleep_for(std::chrono::milliseconds(2));
          x.b = 200 + dev;
          ++made[dev];
          return true;
        });
        if (!ok || v.a != 100 + dev || v.b != 200 + dev) ++wrong;
      }
    });
  for (auto& x : threads) x.join();
  for (auto& m : made) std::printf("%d ", m.load());
  tf::PerDevice<Two> u;
  int tries = 0;
  Two v{};
  auto flaky = [&](Two& x) { x.a = 7; return ++tries > 1; };
  const bool first = u.get(1, v, flaky);
  const bool second = u.get(1, v, flaky);
  u.get(1, v, flaky);
  std::printf("%d %d %d %d %lld ", wrong.load(), first, second, tries, v.a);
  int big = 0;                                    // beyond the table: still made, each time
  for (int i = 0; i < 2; ++i) u.get(1000, v, [&](Two& x) { x.a = ++big; return true; });
  std::printf("%lld\n", v.a);
}
"""


def test_set_up_is_made_once_per_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "p")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", CSRC, "-o", exe, str(tmp_path / "p.cpp")],
                   check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == \
        "1 1 1 1 0 0 1 2 7 2".split()


@pytest.mark.parametrize("name", ["tf_thread.cuh", "tf_rows.cuh"])
def test_launches_keep_their_set_up_per_device(name):
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert not re.findall(r"^\s+static (?:int|bool|long long)\b[^(;]*[=\[;]", code, flags=re.M)
    assert "static PerDevice<" in code
