"""Compile the CUDA library ``libtontofock.so`` for sm_100a (in-tree).

    python -m tonto_b200.build

The library is written next to this file so that it travels with the source tree.

A process loads a source's kernels when it first launches one of them, in time that goes with
their size: with line tables the library unpacks to 177 MB, without to 53 MB.  So line tables
are built in only when asked for (TF_LINEINFO=1 with --force, for a profile by source line),
and the kernels are stored unpacked.  Measured in fresh processes, median ms of context
creation and first build, line tables (packed) -> neither: (H2O)2 cc-pVDZ 17.3 + 83.8 ->
8.0 + 15.6; minima for (H2O)2 STO-3G 61 -> 17, (H2O)2 cc-pVTZ 139 -> 35.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtontofock.so")
PEAK_LIB = os.path.join(HERE, "libtf_peak.so")

SOURCES = ["tontofock.cu", "tf_jk_ss.cu", "tf_jk_ps.cu", "tf_jk_d.cu", "tf_jk_f.cu", "tf_jk_l.cu", "tf_jk_l2.cu", "tf_rows_d.cu",
           "tf_rows_fs.cu", "tf_rows_fd.cu", "tf_rows_ff.cu", "tf_mlp.cu"]
DEPS = SOURCES + ["tf_device.cuh", "tf_thread.cuh", "tf_rows.cuh", "tf_warp.cuh", "tf_host.h", "rys_tables.inc", "boys_table.inc", "boys2_table.inc",
        os.path.join("..", "build.py"), os.path.join("..", "..", "include", "tontofock.h"), os.path.join("..", "..", "include", "tontofock_guess.h")]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def flags() -> list:
    lineinfo = ["-lineinfo"] if os.environ.get("TF_LINEINFO", "0") != "0" else []
    return ["-gencode", "arch=compute_100a,code=sm_100a", *lineinfo, "--compress-mode=none", "-O3", "-std=c++17",
            "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared"]


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(os.path.join(CSRC, d)) <= t for d in DEPS)


def build_peak(force: bool = False) -> str:
    src = os.path.join(CSRC, "fp64_peak.cu")
    if force or not os.path.exists(PEAK_LIB) or os.path.getmtime(src) > os.path.getmtime(PEAK_LIB):
        subprocess.run([nvcc()] + flags() + ["-o", PEAK_LIB, src], check=True, cwd=CSRC)
    return PEAK_LIB


def build(force: bool = False, verbose: bool = False) -> str:
    build_peak(force)
    if not force and up_to_date():
        return LIB
    # one object per source, compiled side by side: the kernels are split over the
    # sources by angular momentum so that they are
    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, src + ".o") for src in SOURCES]

        def compile_one(src: str, obj: str) -> None:
            cmd = [nvcc()] + [f for f in flags() if f != "-shared"] + ["-c", "-o", obj, os.path.join(CSRC, src)]
            if verbose:
                print(" ".join(cmd), flush=True)
            subprocess.run(cmd, check=True, cwd=CSRC)

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            list(pool.map(compile_one, SOURCES, objs))
        subprocess.run([nvcc()] + flags() + ["-o", LIB + ".tmp"] + objs, check=True, cwd=CSRC)
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
