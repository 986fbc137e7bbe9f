"""Large calls let the next one be set up before they end, and it fetches its sources ahead: whatever the calls in a row
read of one another's results, and write over one another's sources, comes out as in stream order."""
import pytest
import torch

from allreduce_over_mpi_b200.ops import HostReducePipeline, reduce_nway, reduce_nway_scaled
from allreduce_over_mpi_b200.parallel.comm import LocalWorld

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
N = 5_000_011   # three int32 vectors in, one out: 80 MB


def vectors(n, offsets, dtype=torch.int32, seed=1):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randint(-1000, 1000, (N + o,), generator=g, device=DEV).to(dtype)[o:] for _, o in zip(range(n), offsets)]


@pytest.mark.parametrize("offsets", [(0, 0, 0, 0), (1, 1, 1, 0), (0, 1, 2, 3)], ids=["wide", "realign", "shift"])
@pytest.mark.parametrize("between", ["nothing", "small", "torch"])
def test_chain_of_sums(offsets, between):
    ring, want = vectors(4, offsets), vectors(4, offsets)
    tiny = [torch.ones(64, dtype=torch.int32, device=DEV) for _ in range(2)]
    for step in range(16):   # each result is a source of the next call, over the oldest source of this one
        k = [(step + j) % 4 for j in range(4)]
        reduce_nway([ring[k[0]], ring[k[1]], ring[k[2]]], out=ring[k[3]])
        if between == "small":
            reduce_nway(tiny, out=tiny[step % 2])
        elif between == "torch":
            ring[k[3]].add_(step)
    torch.cuda.synchronize()
    for step in range(16):
        k = [(step + j) % 4 for j in range(4)]
        want[k[3]].copy_(want[k[0]] + want[k[1]] + want[k[2]] + (step if between == "torch" else 0))
        torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(ring, want))


def test_chain_of_averages():
    ring = vectors(4, (0, 0, 0, 0), torch.float32)
    want = [v.clone() for v in ring]
    for step in range(12):
        k = [(step + j) % 4 for j in range(4)]
        reduce_nway_scaled([ring[k[0]], ring[k[1]], ring[k[2]]], scale=0.5, out=ring[k[3]])
    torch.cuda.synchronize()
    for step in range(12):
        k = [(step + j) % 4 for j in range(4)]
        want[k[3]].copy_((want[k[0]] + want[k[1]] + want[k[2]]) * 0.5)   # the kernel's additions, in its order
    assert all(torch.equal(a, b) for a, b in zip(ring, want))


@pytest.mark.parametrize("shape", ["2", "4", "2*4"])
def test_chain_of_collectives(shape):
    world = {"2": 2, "4": 4, "2*4": 8}[shape]
    count = (64 << 20) // 4 // world + 5
    w = LocalWorld(world, heap_bytes=(count * 4 + (1 << 20)), staging_bytes=1 << 20)
    ts = [c.alloc(count, torch.int32) for c in w.ranks]
    g = torch.Generator(device=DEV).manual_seed(3)
    host = [torch.randint(-1000, 1000, (count,), generator=g, device=DEV).to(torch.int32) for _ in ts]
    for t, h in zip(ts, host):
        t.copy_(h)
    want = torch.stack(host).sum(0, dtype=torch.int32)
    for step in range(6):   # every rank's copy is the sum of all, so each call multiplies by the world
        w.all_reduce(ts, shape=shape)
        w.reduce_scatter(ts, shape=shape)
        w.all_gather(ts, shape=shape)
    torch.cuda.synchronize()
    want = want * (world ** 11 % (1 << 32) if world ** 11 % (1 << 32) < 1 << 31 else world ** 11 % (1 << 32) - (1 << 32))
    assert all(torch.equal(t, want) for t in ts)
    w.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", ["2", "4", "2*4", "2*2*2"])
@pytest.mark.parametrize("copies", [64 << 20, 110 << 20], ids=["64MB", "110MB"])
def test_chain_of_float_collectives(shape, dtype, copies):
    """As above on the compiled programs, with the halves' choice of what leaves L2 for copies that it holds and that it does
    not, and a reader behind the gather.  Small whole numbers times a power of two: exact, whatever the order."""
    world = {"2": 2, "4": 4, "2*4": 8, "2*2*2": 8}[shape]
    count = copies // dtype.itemsize // world + 5
    w = LocalWorld(world, heap_bytes=count * dtype.itemsize + (1 << 20), staging_bytes=1 << 20)
    ts = [c.alloc(count, dtype) for c in w.ranks]
    g = torch.Generator(device=DEV).manual_seed(3)
    want = torch.zeros(count, device=DEV)
    for t in ts:
        h = torch.randint(-8, 8, (count,), generator=g, device=DEV).to(dtype)
        t.copy_(h)
        want += h.float()
    read = []
    for step in range(4):   # every rank's copy is the sum of all, so each call multiplies by the world
        w.all_reduce(ts, shape=shape)
        owned = w.reduce_scatter(ts, shape=shape)
        for blocks in owned:
            for b in blocks if isinstance(blocks, (list, tuple)) else [blocks]:
                b.mul_(0.5)
        w.all_gather(ts, shape=shape)
        read.append(reduce_nway(ts[:2]))
    torch.cuda.synchronize()
    for step in range(4):
        want *= world * 0.5 * (world if step else 1)
        assert torch.equal(read[step].float(), want * 2)
    assert all(torch.equal(t.float(), want) for t in ts)
    w.close()


def test_two_streams():
    """Each stream's chain for itself, both at once."""
    a, b = vectors(4, (0, 0, 0, 0), seed=5), vectors(4, (0, 0, 0, 0), seed=6)
    want = [[v.clone() for v in a], [v.clone() for v in b]]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for step in range(16):
        k = [(step + j) % 4 for j in range(4)]
        for ring, st in ((a, streams[0]), (b, streams[1])):
            with torch.cuda.stream(st):
                reduce_nway([ring[k[0]], ring[k[1]], ring[k[2]]], out=ring[k[3]])
    torch.cuda.synchronize()
    for ring in want:
        for step in range(16):
            k = [(step + j) % 4 for j in range(4)]
            ring[k[3]].copy_(ring[k[0]] + ring[k[1]] + ring[k[2]])
    assert all(torch.equal(x, y) for x, y in zip(a + b, want[0] + want[1]))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float64, torch.uint8, torch.int64])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 11, 16])
def test_large_calls_of_every_fan_in(n, dtype):
    """Just below and above the size from which calls fetch ahead, ragged at both ends: every element once, none beside."""
    es = dtype.itemsize
    for moved in ((50 << 20) - 4096, (50 << 20) + 8192):
        for head, tail in ((0, 0), (1, 3)):
            length = moved // ((n + 1) * es) // 32 * 32 + (32 - head if head else 0) + tail
            g = torch.Generator(device=DEV).manual_seed(length)
            ts = [torch.randint(0, 20, (length + head,), generator=g, device=DEV).to(dtype)[head:] for _ in range(n)]
            flat = torch.full((length + head + 64,), 99, dtype=dtype, device=DEV)
            out = reduce_nway(ts, out=flat[head:length + head])
            want = ts[0].clone()
            for t in ts[1:]:   # small whole numbers: exact in every type, in any order
                want += t
            assert torch.equal(out, want)
            assert bool((flat[:head] == 99).all()) and bool((flat[length + head:] == 99).all())


@pytest.mark.parametrize("src", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("to", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 16])
def test_large_averages_of_every_fan_in(n, src, to):
    for moved in ((50 << 20) - 8192, (50 << 20) + 16384):
        for head, tail, offset in ((0, 0, 0), (1, 3, 0), (0, 5, 4)):   # offset: results off a 32-byte boundary where that is 16 bytes
            length = moved // (n * src.itemsize + to.itemsize) // 64 * 64 + (32 - head if head else 0) + tail
            g = torch.Generator(device=DEV).manual_seed(length)
            ts = [torch.randint(0, 20, (length + head,), generator=g, device=DEV).to(src)[head:] for _ in range(n)]
            flat = torch.full((length + head + offset + 64,), 99.0, dtype=to, device=DEV)
            out = reduce_nway_scaled(ts, scale=0.5, out=flat[head + offset:length + head + offset])
            want = ts[0].float()
            for t in ts[1:]:   # small whole numbers: the sum is exact, one rounding of the result
                want += t.float()
            assert torch.equal(out, (want * 0.5).to(to))
            assert bool((flat[:head + offset] == 99).all()) and bool((flat[length + head + offset:] == 99).all())


@pytest.mark.parametrize("src", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("to", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [2, 4, 6, 7, 8, 12])
def test_averages_with_edges_of_every_length(n, src, to):
    """The edges are summed by code of their own: from none to a line in front and behind, in calls of both kinds."""
    unit = 32 // src.itemsize
    for body in (3 * unit, (51 << 20) // (n * src.itemsize + to.itemsize)):
        for head, tail in ((0, 1), (1, 0), (unit - 1, unit - 1), (unit // 2, 3), (5, 2 * unit + 1)):
            length = body // unit * unit + head + tail
            g = torch.Generator(device=DEV).manual_seed(length)
            ts = [torch.randint(0, 20, (length + 7,), generator=g, device=DEV).to(src)[7:] for _ in range(n)]
            flat = torch.full((length + 64,), 99.0, dtype=to, device=DEV)
            out = reduce_nway_scaled(ts, scale=0.25, out=flat[7:length + 7])
            want = torch.stack(ts).float().sum(0)   # small whole numbers: the sum is exact, one rounding of the result
            assert torch.equal(out, (want * 0.25).to(to))
            assert bool((flat[:7] == 99).all()) and bool((flat[length + 7:] == 99).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float64, torch.uint8, torch.int64])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 9, 16])
def test_large_realigned_sums(n, dtype):
    """Sources at one offset, the result at another, ragged, just below and above the size from which calls fetch ahead."""
    es = dtype.itemsize
    for moved in ((50 << 20) - 8192, (50 << 20) + 8192, 58 << 20):
        for src, dst, tail in ((1, 0, 0), (0, 1, 5), (16 // es + 1, 2, 1)):
            length = moved // ((n + 1) * es) // 32 * 32 + tail
            g = torch.Generator(device=DEV).manual_seed(length)
            ts = [torch.randint(0, 15, (length + src,), generator=g, device=DEV).to(dtype)[src:] for _ in range(n)]
            flat = torch.full((length + dst + 64,), 99, dtype=dtype, device=DEV)
            out = reduce_nway(ts, out=flat[dst:length + dst])
            want = ts[0].clone()
            for t in ts[1:]:   # small whole numbers: exact in every type, in any order
                want += t
            assert torch.equal(out, want)
            assert bool((flat[:dst] == 99).all()) and bool((flat[length + dst:] == 99).all())


@pytest.mark.parametrize("offsets", [(0, 0, 0, 0), (1, 1, 1, 0)], ids=["wide", "realign"])
def test_chain_in_a_graph(offsets):
    """In a captured graph the request becomes a programmatic edge between the nodes."""
    ring, want = vectors(4, offsets, seed=9), vectors(4, offsets, seed=9)
    stream = torch.cuda.Stream()

    def row(ts, total):
        for step in range(12):
            k = [(step + j) % 4 for j in range(4)]
            total(ts[k[0]], ts[k[1]], ts[k[2]], ts[k[3]])

    with torch.cuda.stream(stream):
        row(vectors(4, offsets), lambda a, b, c, d: reduce_nway([a, b, c], out=d))   # what is made on first use is made
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            row(ring, lambda a, b, c, d: reduce_nway([a, b, c], out=d))
        for _ in range(3):
            graph.replay()
    torch.cuda.synchronize()
    for _ in range(3):
        row(want, lambda a, b, c, d: d.copy_(a + b + c))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(ring, want))


@pytest.mark.parametrize("graph", [False, True], ids=["stream", "graph"])
def test_kernels_that_ask_one_after_the_other(graph):
    """Every kernel that asks early in front of and behind the others, the host's vectors among them: sums, sums off the
    sources' boundary, averages, and the collectives' programs and copies, each reading what the one before it wrote."""
    world = LocalWorld(4, heap_bytes=N * 4 + (1 << 20), staging_bytes=1 << 20)
    ts = [c.alloc(N, torch.float32) for c in world.ranks]
    host = [torch.randint(0, 9, (70_001,)).float().pin_memory() for _ in range(3)]
    out = torch.empty(70_001).pin_memory()
    pipe = HostReducePipeline(device=DEV, max_inputs=3, max_outputs=1)

    def start():
        g = torch.Generator(device=DEV).manual_seed(2)
        return [torch.randint(-4, 5, (N,), generator=g, device=DEV).float() for _ in range(10)]

    def row(v, total, average, collective, half, hosts):   # values stay below 2^22 of their smallest step: exact in any order
        a, b, c, d, e, f = v[:6]
        for _ in range(2):
            total([a, b, c], d)
            total([d[1:], b[1:]], e[:-1])
            average([d, e, a], 0.5, f)
            total([f, d], v[6])
            collective(v[6:])
            half(v[6:])
            hosts()
            total([v[6], v[9], f], a)
            average([a, d], 0.25, b)

    def ours(v):
        row(v, lambda x, o: reduce_nway(x, out=o), lambda x, s, o: reduce_nway_scaled(x, scale=s, out=o),
            lambda x: world.all_reduce(x, shape="2*2"), lambda x: (world.reduce_scatter(x, shape="4"), world.all_gather(x, shape="4")),
            lambda: pipe.run(host, [3], [out]))

    def summed(x):
        s = x[0] + x[1] + x[2] + x[3]
        for t in x:
            t.copy_(s)

    got, want = start(), start()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        mine = got[:6] + ts
        if graph:
            for t, h in zip(ts, got[6:]):
                t.copy_(h)
            ours([v.clone() for v in got[:6]] + ts)   # what is made on first use is made
            stream.synchronize()
            recorded = torch.cuda.CUDAGraph()
            with torch.cuda.graph(recorded, stream=stream):
                ours(mine)
        for t, h in zip(ts, got[6:]):
            t.copy_(h)
        if graph:
            recorded.replay()
        else:
            ours(mine)
    torch.cuda.synchronize()
    row(want, lambda x, o: o.copy_(sum(x[1:], x[0])), lambda x, s, o: o.copy_(sum(x[1:], x[0]) * s), summed, summed, lambda: None)
    assert all(torch.equal(x, y) for x, y in zip(mine, want))
    assert torch.equal(out, host[0] + host[1] + host[2])
    world.close()
    pipe.close()
