"""The library's first use in a process costs what its kernels' size costs: line tables, which
tripled it, are built in only when asked for."""

import os

from tonto_b200 import build


def test_line_tables_only_when_asked_for(monkeypatch):
    monkeypatch.delenv("TF_LINEINFO", raising=False)
    assert "-lineinfo" not in build.flags()
    monkeypatch.setenv("TF_LINEINFO", "1")
    assert "-lineinfo" in build.flags()


def test_library_size():
    # 53 MB at the time of writing, 177 MB with line tables (both unpacked); a fifth more allowed
    assert os.path.getsize(build.build()) < 64e6
