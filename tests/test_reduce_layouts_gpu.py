"""One-launch n-way reduction over every way vectors can lie: pointers that agree modulo 32 bytes (32-byte kernel with
edges) or not (shifted kernel), at the lengths where body and edges meet."""
import pytest
import torch

from allreduce_over_mpi_b200.ops import launch_count, reduce_nway, reduce_nway_scaled

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENGTHS = [1, 2, 7, 31, 32, 33, 63, 64, 65, 97, 511, 513, 4095, 8193, 100_003]
# offsets in elements: of each source in turn, and of the result
OFFSETS = [((0,), 0), ((1,), 1), ((4,), 4), ((1,), 0), ((0,), 3), ((0, 1, 2, 3), 5), ((7, 0), 2)]


@pytest.mark.parametrize("srcs,dst", OFFSETS)
@pytest.mark.parametrize("dtype,op", [(torch.float32, "sum"), (torch.bfloat16, "sum"), (torch.float16, "sum"), (torch.float64, "sum"),
                                      (torch.int8, "sum"), (torch.int16, "sum"), (torch.int64, "sum"), (torch.int32, "band"),
                                      (torch.uint8, "band"), (torch.bool, "sum")])
def test_every_layout_and_length(dtype, op, srcs, dst):
    for length in LENGTHS:
        for n in (1, 3, 8, 11):
            g = torch.Generator().manual_seed(length * 40 + n)
            host = [torch.randint(0, 2 if dtype == torch.bool else 100, (length + 8,), generator=g).to(dtype) for _ in range(n)]
            ts = [h.to(DEV)[srcs[k % len(srcs)]:][:length] for k, h in enumerate(host)]
            flat = torch.zeros(length + 16, dtype=dtype, device=DEV)
            before = launch_count()
            reduce_nway(ts, op=op, out=flat[dst:dst + length])
            assert launch_count() == before + 1
            want = ts[0].clone()
            for t in ts[1:]:
                want = want & t if op == "band" else want | t if dtype == torch.bool else want + t   # whole numbers: exact in every type
            if dtype == torch.bfloat16:
                want = sum(t.float() for t in ts).to(dtype)
            assert torch.equal(flat[dst:dst + length], want), (length, n)
            assert not flat[:dst].any() and not flat[dst + length:].any()


def test_in_place_with_sources_at_other_phases():
    base = torch.randn(3, 10_020, device=DEV)
    ts = [base[0, 1:10_001], base[1, 2:10_002], base[2, 4:10_004]]
    want = ts[0] + ts[1] + ts[2]
    assert torch.equal(reduce_nway(ts, out=ts[0]), want)
    assert torch.equal(base[0, 1:10_001], want)


@pytest.mark.parametrize("srcs,dst", [((0,), 0), ((3,), 3), ((8,), 0), ((4,), 8), ((0, 1), 0)])
@pytest.mark.parametrize("tin", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tout", [torch.float32, torch.bfloat16])
def test_scaled_every_layout_and_length(tin, tout, srcs, dst):
    """256-bit, 128-bit and one-element forms, with heads and tails; small whole numbers, so every sum is exact."""
    for length in (1, 7, 8, 15, 16, 17, 31, 33, 47, 1000, 4099, 70_001):
        for n in (1, 4, 5, 9):
            g = torch.Generator().manual_seed(length + n)
            ts = [torch.randint(-8, 8, (length + 8,), generator=g).to(tin).to(DEV)[srcs[k % len(srcs)]:][:length] for k in range(n)]
            flat = torch.zeros(length + 16, dtype=tout, device=DEV)
            reduce_nway_scaled(ts, scale=0.25, out=flat[dst:dst + length])
            want = (sum(t.float() for t in ts) * 0.25).to(tout)
            assert torch.equal(flat[dst:dst + length], want), (length, n)
            assert not flat[:dst].any() and not flat[dst + length:].any()
