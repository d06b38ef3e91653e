"""Launches on branch streams: the branches are joined however the scope ends.

tf_host.h takes the runtime calls as a parameter, so this compiles it for the host with a
runtime that logs them, and returns early between fork and join as an allocation or launch
failure would."""

import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tonto_b200", "csrc")

PROGRAM = r"""
#include "tf_host.h"
#include <cstdio>
struct Rt {
  using Stream = int; using Event = int; using Status = int;
  static int fail_at;
  static int next() { return fail_at-- == 0 ? 1 : 0; }
  static int record(int e, int s) { int r = next(); if (!r) std::printf("record %d %d\n", e, s); return r; }
  static int wait(int s, int e) { int r = next(); if (!r) std::printf("wait %d %d\n", s, e); return r; }
};
int Rt::fail_at = -1;
static int scope(int n, bool fails) {
  const std::vector<int> side{1, 2, 3}, ev{11, 12, 13};
  tf::BranchFork<Rt> b(0, side, 10, ev, n);
  if (int r = b.fork()) return r;
  std::printf("launch\n");
  if (fails) return 2;
  return b.join();
}
int main(int argc, char** argv) {
  Rt::fail_at = std::atoi(argv[3]);
  std::printf("rc %d\n", scope(std::atoi(argv[1]), std::atoi(argv[2]) != 0));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fork")
    (d / "fork.cpp").write_text("#include <cstdlib>\n" + PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", str(d / "fork"), str(d / "fork.cpp")],
                   check=True)
    return lambda *a: subprocess.run([str(d / "fork"), *map(str, a)], check=True, capture_output=True,
                                     text=True).stdout.split("\n")[:-1]


@pytest.mark.parametrize("n", [1, 2, 4])
@pytest.mark.parametrize("fails", [0, 1])
def test_branches_are_joined_on_success_and_on_an_early_return(program, n, fails):
    out = program(n, fails, -1)
    want = ["record 10 0"] * (n > 1) + [f"wait {i} 10" for i in range(1, n)] + ["launch"]
    join = [x for i in range(1, n) for x in (f"record {10 + i} {i}", f"wait 0 {10 + i}")]
    rc = [f"rc {2 if fails else 0}"]
    assert [x for x in out if not x.startswith("rc")] == want + join and [x for x in out if x.startswith("rc")] == rc


def test_a_fork_that_fails_half_way_joins_what_it_forked(program):
    # the second branch's wait fails: the first branch, already waiting, is joined
    assert program(4, 0, 2) == ["record 10 0", "wait 1 10", "record 11 1", "wait 0 11", "rc 1"]


def test_the_library_forks_through_the_guard_only():
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "tontofock.cu")).read())
    uses = re.findall(r"cudaEventRecord\s*\(\s*c->(fork_ev|join_ev)", code)
    assert not uses and len(re.findall(r"\bFork \w+\(c, ", code)) >= 4
