"""The entry points where the native call path (lib/_ft_torch-*.so) cannot be built or loaded: the same results, through
Python and ctypes, after one warning.  Each case is a process of its own, since a process looks for it once."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
HEAD = """
import warnings, torch
from pathlib import Path
from allreduce_over_mpi_b200 import _lib, build
tmp = Path(%r)
build.LIB = tmp / "libflextree.so"           # where the call path is looked for; the library itself stays where it is
with warnings.catch_warnings(record=True) as said:
    warnings.simplefilter("always")
    _lib.native()
    _lib.native()
assert len(said) == 1 and "no native call path" in str(said[0].message), [str(s.message) for s in said]
"""


def run(tmp_path, monkeypatch, cxx, code):
    monkeypatch.setenv("CXX", cxx)
    r = subprocess.run([sys.executable, "-c", HEAD % str(tmp_path) + code], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, (r.stdout[-1000:], r.stderr[-3000:])


def compiler(tmp_path, kind):
    if kind == "none":
        return str(tmp_path / "no-such-compiler")
    if kind == "fails":                      # e.g. no Python.h
        return "/bin/false"
    path = tmp_path / "cxx"                  # what it makes cannot be loaded, as with libraries of another torch
    path.write_text(f"#!{sys.executable}\nimport sys\nopen(sys.argv[sys.argv.index('-o') + 1], 'w').write('no library')\n")
    path.chmod(0o755)
    return str(path)


@pytest.mark.parametrize("kind", ["none", "fails", "unloadable"])
def test_cpu_tensors_are_reduced(tmp_path, monkeypatch, kind):
    run(tmp_path, monkeypatch, compiler(tmp_path, kind), """
from allreduce_over_mpi_b200.ops import cpu_reduce, reduce_nway, reduce_nway_scaled
ts = [torch.full((1001,), float(k)) for k in range(5)]
out = torch.empty(1001)
assert reduce_nway(ts, out=out) is out and bool((out == 10).all()) and bool((cpu_reduce(ts) == 10).all())
assert reduce_nway([torch.tensor([6, 3]), torch.tensor([3, 5])], op="band").tolist() == [2, 1]
try:
    reduce_nway_scaled(ts)
except ValueError as e:
    assert "device" in str(e)
else:
    raise AssertionError
""")


@pytest.mark.gpu
def test_cuda_tensors_are_reduced(tmp_path, monkeypatch):
    run(tmp_path, monkeypatch, compiler(tmp_path, "none"), """
from allreduce_over_mpi_b200.ops import HostReducePipeline, launch_count, reduce_nway, reduce_nway_scaled
from allreduce_over_mpi_b200.parallel.comm import LocalWorld
ts = [torch.full((1001,), float(k), device="cuda") for k in range(4)]
assert bool((reduce_nway(ts) == 6).all()) and launch_count() == 1
assert bool((reduce_nway_scaled(ts, scale=0.5, out_dtype=torch.bfloat16) == 3).all()) and launch_count() == 2
pin = [t.cpu().pin_memory() for t in ts]
outs = [torch.empty(1001).pin_memory() for _ in range(2)]
pipe = HostReducePipeline(device="cuda:0", max_inputs=4, max_outputs=2)
pipe.run(pin, [2, 4], outs)
torch.cuda.synchronize()
assert bool((outs[0] == 1).all()) and bool((outs[1] == 6).all())
pipe.close()
w = LocalWorld(4, heap_bytes=1 << 20, staging_bytes=1 << 20)
w.all_reduce(ts, shape="2*2")
heap = [c.alloc(1001).fill_(float(c.rank)) for c in w.ranks]
owned = w.reduce_scatter(heap, shape="2*2")
torch.cuda.synchronize()
assert all(bool((t == 6).all()) for t in ts) and all(bool((v == 6).all()) for views in owned for v in views)
assert sum(v.numel() for views in owned for v in views) == 1001
w.close()
""")
