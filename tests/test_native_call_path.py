"""The native call path of the Python entry points (csrc/python/ft_torch.cpp), as far as a CPU takes it: whatever it
cannot take it hands back (NotImplemented) or reports as a Python exception; it never takes the interpreter down.
What used to end the process runs in a child."""
import subprocess
import sys
from pathlib import Path

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
