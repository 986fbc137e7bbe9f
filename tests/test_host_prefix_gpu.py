"""Prefix reductions of host vectors: pinned and aligned (one kernel over PCIe) or not (chunked copies), same results."""
import pytest
import torch

from allreduce_over_mpi_b200.ops import HostReducePipeline, launch_count, reduce_nway

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,op", [(torch.float32, "sum"), (torch.bfloat16, "sum"), (torch.float64, "sum"), (torch.int16, "sum"),
                                      (torch.uint8, "band"), (torch.int64, "band")])
@pytest.mark.parametrize("n,fanins", [(1, [1]), (8, [2, 3, 4, 8]), (9, [9, 1, 9]), (12, [5])])
def test_pinned_pageable_and_unaligned(dtype, op, n, fanins):
    for length in (1, 15, 4099, 70_003):
        g = torch.Generator().manual_seed(length)
        vecs = [torch.randint(0, 100, (length,), generator=g).to(dtype) for _ in range(n)]
        want = [reduce_nway([v.to(DEV) for v in vecs[:f]], op=op).cpu() for f in fanins]
        pipe = HostReducePipeline(device=DEV, chunk_bytes=64 << 10, max_inputs=n, max_outputs=len(fanins))
        for kind in ("pinned", "pageable", "unaligned", "mixed"):
            pin = kind in ("pinned", "unaligned")
            off = 1 if kind == "unaligned" else 0
            hin = [torch.empty(length + off, dtype=dtype, pin_memory=pin or (kind == "mixed" and k == 0))[off:].copy_(v) for k, v in enumerate(vecs)]
            flat = [torch.zeros(length + 16 + off, dtype=dtype, pin_memory=pin) for _ in fanins]
            outs = [f[off:length + off] for f in flat]
            before = launch_count()
            pipe.run(hin, fanins, outs, op=op)
            torch.cuda.synchronize()
            assert all(torch.equal(o, w) for o, w in zip(outs, want)), (kind, length)
            assert not any(f[length + off:].any() for f in flat)
            if kind == "pinned":
                assert launch_count() == before + 1
        pipe.close()


def test_in_place_and_own_stream():
    hin = [torch.randn(100_003).pin_memory() for _ in range(3)]
    want = (hin[0].to(DEV) + hin[1].to(DEV) + hin[2].to(DEV)).cpu()
    pipe = HostReducePipeline(device=DEV, max_inputs=3, max_outputs=1)
    st = torch.cuda.Stream()
    pipe.run(hin, [3], [hin[1]], stream=st)
    st.synchronize()
    assert torch.equal(hin[1], want)
    pipe.close()


def test_results_over_later_inputs_and_over_one_another():
    """Every input of a chunk is read before any result is written, and the last of two results in one place stays."""
    host = [torch.randn(5003) for _ in range(12)]
    hin = [h.pin_memory() for h in host]
    want = [reduce_nway([h.to(DEV) for h in host[:f]]).cpu() for f in (5, 12, 3)]
    pipe = HostReducePipeline(device=DEV, max_inputs=12, max_outputs=3)
    both = torch.empty(5003).pin_memory()
    pipe.run(hin, [5, 12, 3], [hin[10], both, both])
    torch.cuda.synchronize()
    assert torch.equal(hin[10], want[0]) and torch.equal(both, want[2])
    pipe.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.uint8])
@pytest.mark.parametrize("n", [2, 3, 8])
def test_cuts_of_the_pcie_kernel(dtype, n):
    """Around a CTA's vectors, a warp of vectors with elements behind it, and the step to two vectors a thread: a last turn
    that is full, nearly empty, or elements only."""
    es = dtype.itemsize
    pipe = HostReducePipeline(device=DEV, max_inputs=n, max_outputs=2)
    for nvec in (0, 1, 31, 32, 1023, 1024, 6144, 6145, 18_432, 18_433, 24_577):
        for tail in (0, 1, 16 // es - 1):
            length = nvec * (16 // es) + tail
            if not length:
                continue
            g = torch.Generator().manual_seed(length)
            vecs = [torch.randint(0, 100, (length,), generator=g).to(dtype).pin_memory() for _ in range(n)]
            flat = [torch.zeros(length + 32, dtype=dtype, pin_memory=True) for _ in range(2)]
            pipe.run(vecs, [1, n], [f[:length] for f in flat])
            torch.cuda.synchronize()
            assert torch.equal(flat[0][:length], vecs[0])
            assert torch.equal(flat[1][:length], reduce_nway([v.to(DEV) for v in vecs]).cpu()), (nvec, tail)
            assert not any(f[length:].any() for f in flat)
    pipe.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.uint8])
@pytest.mark.parametrize("n", [1, 2, 4, 5])
def test_two_vectors_a_thread_in_one_cta(dtype, n):
    """Between one and two vectors for each thread of a CTA: the second ones from none to all, with elements behind them, in
    place too."""
    per = 16 // dtype.itemsize
    pipe = HostReducePipeline(device=DEV, max_inputs=n, max_outputs=2)
    for nvec in (1024, 1025, 1055, 1056, 1057, 1536, 2015, 2016, 2017, 2047, 2048):
        for tail in (0, 1, per - 1):
            length = nvec * per + tail
            g = torch.Generator().manual_seed(length)
            vecs = [torch.randint(0, 25, (length,), generator=g).to(dtype).pin_memory() for _ in range(n)]
            want = [reduce_nway([v.to(DEV) for v in vecs[:f]]).cpu() for f in (1, n)]
            flat = torch.zeros(length + 32, dtype=dtype, pin_memory=True)
            pipe.run(vecs, [1, n], [flat[:length], vecs[n - 1]])
            torch.cuda.synchronize()
            assert torch.equal(flat[:length], want[0]) and torch.equal(vecs[n - 1], want[1]), (nvec, tail)
            assert not flat[length:].any()
    pipe.close()
