"""When and how the native call path is compiled: a compiler that only writes a file stands in for g++."""
import os
import subprocess
import sys
import time
from pathlib import Path

import pytest

from allreduce_over_mpi_b200 import build

ROOT = Path(__file__).resolve().parents[1]
FAKE = """#!%s
import os, sys, time
open(os.environ["FAKE_LOG"], "a").write("run\\n")
if os.environ.get("FAKE_FAIL"):
    sys.exit("no such header")
with open(sys.argv[sys.argv.index("-o") + 1], "w") as f:
    f.write("first half,"); f.flush(); time.sleep(0.5); f.write("second half")
""" % sys.executable


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A library folder and sources of their own, and the compiler above; returns how often it ran so far."""
    cxx, log = tmp_path / "fake_cxx", tmp_path / "log"
    cxx.write_text(FAKE)
    cxx.chmod(0o755)
    log.write_text("")
    src = tmp_path / "ft_torch.cpp", tmp_path / "ft_types.h"
    for s in src:
        s.write_text("// first")
    monkeypatch.setenv("CXX", str(cxx))
    monkeypatch.setenv("FAKE_LOG", str(log))
    monkeypatch.setattr(build, "LIB", tmp_path / "lib" / "libflextree.so")
    monkeypatch.setattr(build, "EXT_SOURCES", src)
    return lambda: len(log.read_text().split())


def test_an_edit_or_another_torch_is_noticed(tree, monkeypatch):
    import torch
    first = build.build_ext()
    assert build.build_ext() == first and tree() == 1
    os.utime(build.EXT_SOURCES[0])                          # touched, not edited
    assert build.build_ext() == first and tree() == 1
    build.EXT_SOURCES[1].write_text("// second")
    edited = build.build_ext()
    assert edited != first and tree() == 2 and not first.exists()
    monkeypatch.setattr(torch, "__version__", "99.0")
    other = build.build_ext()
    assert other != edited and tree() == 3 and edited.exists()   # both stay: each torch finds its own


def test_a_failed_compiler_leaves_nothing_behind(tree, monkeypatch):
    monkeypatch.setenv("FAKE_FAIL", "1")
    with pytest.raises(RuntimeError, match="no such header"):
        build.build_ext()
    assert [p.name for p in build.LIB.parent.iterdir()] == [".build.lock"]


def test_ranks_started_together_compile_once_and_never_see_half_a_file(tree):
    code = (f"from pathlib import Path\nfrom allreduce_over_mpi_b200 import build\nbuild.LIB = Path({str(build.LIB)!r})\n"
            f"build.EXT_SOURCES = tuple(map(Path, {list(map(str, build.EXT_SOURCES))!r}))\n"
            "import torch\nprint('up', flush=True)\ninput()\nprint(build.build_ext().read_text())")
    ranks = [subprocess.Popen([sys.executable, "-c", code], stdin=subprocess.PIPE, stdout=subprocess.PIPE, text=True, cwd=ROOT) for _ in range(3)]
    try:
        for p in ranks:
            assert p.stdout.readline().strip() == "up"
        for p in ranks:
            p.stdin.write("\n")
            p.stdin.flush()
        ext, deadline = build.ext_path(), time.time() + 60
        while not ext.exists() and time.time() < deadline:
            time.sleep(0.01)
        assert ext.read_text() == "first half,second half"
        assert [p.communicate(timeout=60)[0].strip() for p in ranks] == ["first half,second half"] * 3
    finally:
        for p in ranks:
            p.kill()
    assert tree() == 1
