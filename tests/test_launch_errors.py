"""A launch that the runtime refuses is reported once, by the call it belongs to, and is not counted as a launch."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def child(code, **env):
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=300, env={**os.environ, **env})
    assert r.returncode == 0, (r.stdout[-1000:], r.stderr[-3000:])
    return r.stdout.strip()


def test_refused_launches_are_not_counted():
    """With no device to be seen every launch is refused; ordinary host memory stands in for the vectors."""
    assert child("""
import ctypes as C
from allreduce_over_mpi_b200._lib import lib
L = lib()
bufs = [C.create_string_buffer(8192) for _ in range(4)]
src = (C.c_void_p * 3)(*[C.addressof(b) for b in bufs[:3]])
dst = C.c_void_p(C.addressof(bufs[3]))
codes = [L.ft_reduce_nway(0, 6, src, dst, 3, 1000, variant, None) for variant in (0, 1, 2, 13, 24)]
codes += [L.ft_reduce_nway(0, 6, src, C.c_void_p(dst.value + 4), 3, 1000, 0, None), L.ft_reduce_nway_scaled(6, 11, src, dst, 3, 1000, 0.5, None),
          L.ft_scale_inplace(6, dst, 1000, 0.5, None)]
print(set(codes), L.ft_launch_count(), b"launch" in L.ft_last_cuda_error())
""", CUDA_VISIBLE_DEVICES="") == "{6} 0 True"


@pytest.mark.gpu
def test_a_refused_launch_is_not_reported_by_the_next_one():
    """The stream's capture is void (it was asked to synchronise), so launches on it are refused, on the host.  The calls
    behind it, on another stream, ask the runtime for its last error: it must not be that one."""
    assert child("""
import torch
from allreduce_over_mpi_b200._lib import lib
from allreduce_over_mpi_b200.ops import HostReducePipeline, launch_count, reduce_nway, reduce_nway_scaled
from allreduce_over_mpi_b200.parallel.comm import LocalWorld
ts = [torch.ones(4096, device="cuda") for _ in range(3)]
out = torch.empty_like(ts[0])
pin = [torch.ones(4096).pin_memory() for _ in range(3)]
pipe = HostReducePipeline(device="cuda:0", max_inputs=2, max_outputs=1)
w = LocalWorld(2, heap_bytes=1 << 20, staging_bytes=1 << 20)
reduce_nway(ts, out=out, variant=13)            # everything set up
torch.cuda.synchronize()
calls = {"wide": lambda: reduce_nway(ts, out=out), "shift": lambda: reduce_nway([t[1:] for t in ts], out=out[:-1]),
         "scaled": lambda: reduce_nway_scaled(ts, 0.5, out=out), "host": lambda: pipe.run(pin[:2], [2], pin[2:]),
         "world": lambda: w.all_reduce(ts[:2], shape="2")}
for name, call in calls.items():
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    before = launch_count()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        try:
            s.synchronize()
        except RuntimeError:
            pass
        try:
            call()
        except RuntimeError as e:
            assert "CUDA error" in str(e) and ("captur" in str(e) or "captur" in lib().ft_last_cuda_error().decode()), (name, str(e))
        else:
            raise AssertionError(name)
        try:
            g.capture_end()
        except RuntimeError:
            pass
    assert launch_count() == before, name
    reduce_nway(ts, out=out, variant=13)        # asks for the last error behind its launch
    torch.cuda.synchronize()
    assert bool((out == 3).all()) and launch_count() == before + 1, name
print("ok")
""") == "ok"
