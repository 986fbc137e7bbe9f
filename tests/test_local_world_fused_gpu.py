"""A world on one device: the one-launch form against the kernels that several devices would run.

The tests of test_comm_emulated_gpu.py, and those of test_y_comm_extras_gpu.py on worlds of several ranks, call whatever
``LocalWorld`` runs by default, the one-launch form; they are collected here a second time with it switched off, so that
the multi-GPU kernels stay covered on one GPU: their sums, the guard blocks behind the tensors they write, and the
stage ranges of the two halves (everything a rank does not own is NaN before the gather)."""
import pytest
import torch

import test_comm_emulated_gpu as emulated
import test_y_comm_extras_gpu as extras
from allreduce_over_mpi_b200.ops import launch_count
from allreduce_over_mpi_b200.parallel.comm import LocalWorld
from allreduce_over_mpi_b200.parallel.planner import Shape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class TestStageByStage:
    @pytest.fixture(autouse=True)
    def unfused(self, monkeypatch):
        def refuse(*_):
            raise AssertionError("the one-launch form was asked")
        monkeypatch.setattr(LocalWorld, "fused", False)
        monkeypatch.setattr(LocalWorld, "_run_fused", refuse)

    for _name in dir(emulated):
        if _name.startswith("test_"):
            locals()[_name] = staticmethod(getattr(emulated, _name))
    for _name in ("test_reduce_scatter_and_all_gather_alone", "test_phases_refuse_tensors_outside_the_heap",
                  "test_guard_blocks_behind_heap_tensors_stay_intact", "test_unaligned_slice_of_a_heap_tensor_goes_through_the_slots",
                  "test_heap_free_and_reuse"):
        locals()[_name] = staticmethod(getattr(extras, _name))


def both(world, make, call):
    """The results of `call(world, tensors)` with and without the one-launch form, and how many launches it took."""
    got = []
    for fused in (True, False):
        w = LocalWorld(world, heap_bytes=4 << 20, staging_bytes=4 << 20)
        w.fused = fused
        ts = make(w)
        before = launch_count()
        res = call(w, ts)
        torch.cuda.synchronize()
        got.append(([t.clone() for t in res], launch_count() - before))
        w.close()
    (a, launches), (b, _) = got
    assert all(torch.equal(x.view(torch.uint8), y.view(torch.uint8)) for x, y in zip(a, b))
    return launches


def tensors(world, count, dtype, heap):
    def make(w):
        g = torch.Generator(device=DEV).manual_seed(count)
        out = []
        for c in w.ranks:
            x = (torch.randn(count, generator=g, device=DEV) * 20).to(dtype)
            out.append(c.alloc(count, dtype).copy_(x) if heap else x)
        return out
    return make


@pytest.mark.parametrize("text", emulated.SHAPES + ["ring16", "2*2*2*2"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_every_shape_same_bits(text, dtype):
    n = Shape.parse(text).world
    for count in (35, 4099, 600_000):
        for heap in (False, True):
            make = tensors(n, count, dtype, heap)
            assert both(n, make, lambda w, ts: w.all_reduce(ts, op="avg", shape=text)) == 1
            if heap:
                assert both(n, make, lambda w, ts: (w.reduce_scatter(ts, op="avg", shape=text), ts)[1]) == 1
                assert both(n, make, lambda w, ts: w.all_gather(ts, shape=text)) == 1
            elif count <= 4099:
                assert both(n, make, lambda w, ts: w.all_reduce(ts, shape=text, algo="ll", outs=[torch.empty_like(t) for t in ts])) == 1


@pytest.mark.parametrize("text", ["2", "3", "5", "7", "2*2", "3*2", "4*2", "2*2*2", "ring3", "ring6", "2*2+1", "3*2+1", "2*3+2"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float64, torch.int64, torch.uint8])
def test_compiled_programs_same_bits(text, dtype):
    """Types with a dispatch of their own, around an empty block, a lone element, the step to 32 bytes a thread and, for
    eight ranks, the one from which the halves say what leaves L2 first."""
    n = Shape.parse(text).world
    op = "avg" if dtype.is_floating_point else "sum"
    for count in (1, 8 * n + 1, (2 << 20) // dtype.itemsize - 1, (2 << 20) // dtype.itemsize + 17, (4 << 20) // dtype.itemsize):
        make = tensors(n, count, dtype, True)
        assert both(n, make, lambda w, ts: w.all_reduce(ts, op=op, shape=text)) == 1
        assert both(n, make, lambda w, ts: (w.reduce_scatter(ts, op=op, shape=text), ts)[1]) == 1
        assert both(n, make, lambda w, ts: w.all_gather(ts, shape=text)) == 1


@pytest.mark.parametrize("algo", ["oneshot", "ll", "push"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float64, torch.int64, torch.uint8])
def test_flat_algorithms_same_bits(algo, dtype):
    for world in (2, 7, 8, 11):
        for count in (1, 20_001):
            make = tensors(world, count, dtype, algo == "push")
            assert both(world, make, lambda w, ts: w.all_reduce(ts, op="avg" if dtype.is_floating_point else "sum", algo=algo)) == 1


def test_calls_it_does_not_take_go_stage_by_stage():
    base = torch.randn(4, 2048, device=DEV)
    shifted = lambda w: [b[1:2000] for b in base.clone()]   # noqa: E731 - off a 16-byte boundary
    assert both(4, shifted, lambda w, ts: w.all_reduce(ts, shape="2*2")) > 1

    def overlapping(w):   # rank 1's result starts inside rank 0's input
        flat = base.clone().view(-1)
        return [flat[0:1024], flat[2048:3072], flat[512:1536], flat[4096:5120]]
    assert both(2, overlapping, lambda w, ts: w.all_reduce(ts[:2], shape="2", outs=ts[2:])) > 1
    w = LocalWorld(2, heap_bytes=1 << 20, staging_bytes=1 << 20)
    w.ranks[1].close()
    with pytest.raises(Exception):
        w.all_reduce([base[0], base[1]], shape="2")
    w.close()
