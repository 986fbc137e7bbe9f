"""The native call path of the Python entry points (csrc/python/ft_torch.cpp), as far as a CPU takes it: whatever it
cannot take it hands back (NotImplemented) or reports as a Python exception; it never takes the interpreter down.
What used to end the process runs in a child."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def child(code: str) -> str:
    head = "import torch\nfrom allreduce_over_mpi_b200._lib import native\nN = native()\n"
    r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-3000:])
    return r.stdout.strip()


def test_no_handles_and_no_tensors_are_handed_back():
    """A closed world has no handles; with no tensors either, the counts agree at zero."""
    assert child("""
print(N.local_world_run([], [], [], "sum", (), 0, 0, 0, 0, 1.0), N.local_world_run([], (), (), "sum", (2,), 0, 0, 1, 0, 1.0))
""") == "NotImplemented NotImplemented"


def test_a_closed_world_refuses_an_empty_call():
    assert child("""
from allreduce_over_mpi_b200.parallel.comm import LocalWorld
from allreduce_over_mpi_b200.parallel.planner import Shape
w = LocalWorld.__new__(LocalWorld)      # as after close(): no ranks, no handles
w.world, w.emulated, w.ranks, w._handles, w._flat = 2, True, [], [], Shape.flat(2)
try:
    w.all_reduce([])
except IndexError:
    print("refused")
""") == "refused"


def test_an_exception_in_torch_becomes_a_python_exception():
    """Inside vmap a tensor has no memory: asking for its address throws, in C++."""
    assert child("""
try:
    torch.vmap(lambda x: (N.host_pipe_run(1, 0, [x], [1], [x], "sum"), x)[1])(torch.zeros(2, 3))
except RuntimeError as e:
    print("storage" in str(e))
""") == "True"


def test_narrow_all_reports_what_its_views_raise():
    """A dispatch mode that raises in the second view of the first tensor; without it, the views themselves."""
    assert child("""
from torch.utils._python_dispatch import TorchDispatchMode
class Refuse(TorchDispatchMode):
    calls = 0
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.calls += 1
        if self.calls == 2:
            raise KeyError("no more views")
        return func(*args, **(kwargs or {}))
t = [torch.arange(6.), torch.arange(6.).requires_grad_()]
ranges = (((0, 2), (2, 6)), ((5, 6),))
try:
    with Refuse():
        N.narrow_all(t, ranges)
except KeyError as e:
    print("raised")
v = N.narrow_all(t, ranges)
assert [x.tolist() for x in v[0]] == [[0, 1], [2, 3, 4, 5]] and v[1][0].tolist() == [5]
assert v[0][1]._base is t[0] and not v[0][0].requires_grad and v[1][0].requires_grad
assert N.narrow_all(t, (((0, 7),), ())) is NotImplemented and N.narrow_all([t[0], t[1][:2]], ((), ())) is NotImplemented
""") == "raised"


@pytest.mark.gpu
def test_tensors_of_a_call_outlive_the_lists_they_came_in():
    """While a call runs without the GIL, another thread may change the caller's lists.  The library's entry points are
    replaced by ones that do just that, and look whether the tensors are still there; nothing is launched."""
    assert child("""
import ctypes as C, gc, weakref
from allreduce_over_mpi_b200._lib import _NATIVE
i, sz, vp, f = C.c_int, C.c_size_t, C.c_void_p, C.c_float
sig = {"ft_reduce_nway": (i, i, vp, vp, i, sz, i, vp), "ft_reduce_nway_scaled": (i, i, vp, vp, i, sz, f, vp),
       "ft_local_world_run": (vp, i, vp, vp, sz, i, i, vp, i, i, i, i, i, f, vp),
       "ft_host_pipe_reduce": (vp, i, i, vp, i, vp, vp, i, sz, vp)}
seen = {}
def fake(name):
    def run(*_):
        for l in lists:
            l.clear()
        gc.collect()
        seen[name] = all(w() is not None for w in watched)
        return 0
    return C.CFUNCTYPE(i, *sig[name])(run)
keep = {name: fake(name) for name in _NATIVE}
N.bind({name: C.cast(k, C.c_void_p).value for name, k in keep.items()})
def call(fn, device, count):
    global lists, watched
    lists = [[torch.zeros(64, device=device) for _ in range(2)] for _ in range(count)]
    watched = [weakref.ref(t) for l in lists for t in l]
    fn(*lists)
    assert all(w() is None for w in watched)      # and no longer than the call
call(lambda a: N.reduce_nway(a, "sum", None, 0), "cuda", 1)
call(lambda a: N.reduce_nway_scaled(a, 1.0, None, None), "cuda", 1)
call(lambda a, b: N.local_world_run([1, 2], a, b, "sum", (2,), 0, 0, 1, 0, 1.0), "cuda", 2)
call(lambda a, b: N.host_pipe_run(1, 0, a, [2, 2], b, "sum"), "cpu", 2)
print(sorted(seen) == sorted(_NATIVE) and all(seen.values()))
""") == "True"


@pytest.mark.gpu
def test_a_reduction_inside_vmap_is_refused():
    assert child("""
from allreduce_over_mpi_b200.ops import reduce_nway
try:
    torch.vmap(lambda x: reduce_nway([x, x]))(torch.zeros(2, 8, device="cuda"))
except RuntimeError as e:
    print("storage" in str(e))
""") == "True"
