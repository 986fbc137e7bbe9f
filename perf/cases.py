"""Workloads of the library on one GPU, as a user's program runs them through the public entry points.

``kind`` of a case says which entry point it calls:

* ``nway``    ``ops.reduce_nway``: element-wise reduction of n vectors (gradients of n workers or micro-batches,
              partial results, bit masks);
* ``scaled``  ``ops.reduce_nway_scaled``: gradient averaging with the fp32/bf16 cast fused;
* ``host``    ``ops.HostReducePipeline``: the same reductions for vectors in pinned host memory;
* ``world``   ``LocalWorld.all_reduce``: the collective with every rank on this GPU (replicas that share a device,
              or a plan tried out before it runs on several), by plan, one-shot, tagged words or reduce-and-push;
* ``halves``  ``LocalWorld.reduce_scatter`` then ``all_gather``: what a sharded optimizer does around its update.

``listed`` spans the sizes in use: messages of a few KB (a loss, a norm, the reference's small vectors), the 25 MB
buckets of a data-parallel step, and the 64 Mi-element vectors of ``bench.py``; ``draw`` gives more of the same ranges.
"""
from __future__ import annotations

import math

import torch

from allreduce_over_mpi_b200.ops import HostReducePipeline, reduce_nway, reduce_nway_scaled
from allreduce_over_mpi_b200.parallel.comm import LocalWorld

DEVICE = "cuda:0"
SIZE = {"float32": 4, "float64": 8, "bfloat16": 2, "float16": 2, "int8": 1, "int16": 2, "int32": 4, "int64": 8, "uint8": 1}
FLOATS = ("float32", "float64", "bfloat16", "float16")
BUCKET = 25 << 20   # bytes of a gradient bucket (parallel/ddp.py)


def listed():
    return [
        # a handful of metrics or a small layer's gradient from four workers: all launch latency
        {"name": "nway_f32_x4_4099", "kind": "nway", "dtype": "float32", "op": "sum", "n": 4, "elems": 4099, "offset": 0, "out": False},
        # one ragged layer of bf16 gradients from the eight GPUs of a box
        {"name": "nway_bf16_x8_1M", "kind": "nway", "dtype": "bfloat16", "op": "sum", "n": 8, "elems": 1_000_003, "offset": 0, "out": True},
        # bench.py's vectors
        {"name": "nway_f32_x8_64Mi", "kind": "nway", "dtype": "float32", "op": "sum", "n": 8, "elems": 64 << 20, "offset": 0, "out": True},
        # parameters inside a flat buffer: the slices start wherever the previous parameter ended
        {"name": "nway_f32_x3_views_5M", "kind": "nway", "dtype": "float32", "op": "sum", "n": 3, "elems": 5_000_011, "offset": 1, "out": True},
        # agreement masks (MPI_BAND), the other operation of the library
        {"name": "nway_band_i32_x4_2M", "kind": "nway", "dtype": "int32", "op": "band", "n": 4, "elems": 2_000_003, "offset": 0, "out": False},
        # the widest fan-in of the native n-way benchmark (1..16)
        {"name": "nway_f16_x16_10M", "kind": "nway", "dtype": "float16", "op": "sum", "n": 16, "elems": 10_000_000, "offset": 0, "out": True},
        # average one 25 MB fp32 bucket of eight workers and store it in bf16
        {"name": "scaled_f32_bf16_x8_bucket", "kind": "scaled", "in": "float32", "to": "bfloat16", "n": 8, "elems": BUCKET // 4 + 3,
         "offset": 0},
        # four prefixes of eight host vectors, as bench.py's end-to-end step
        {"name": "host_f32_x8_1Mi", "kind": "host", "dtype": "float32", "n": 8, "fanins": "2,3,4,8", "elems": (1 << 20) + 5},
        # a bf16 gradient bucket averaged in place by a two-level tree
        {"name": "world8_bf16_2x4_bucket", "kind": "world", "algo": "staged", "shape": "2*4", "world": 8, "dtype": "bfloat16",
         "elems": BUCKET // 2, "heap": True},
        # an ordinary fp32 tensor of a few hundred KB, out of place, one-shot
        {"name": "world4_f32_oneshot_100k", "kind": "world", "algo": "oneshot", "shape": "4", "world": 4, "dtype": "float32",
         "elems": 100_001, "heap": False},
        # the smallest collective: a few KB on tagged words
        {"name": "world8_f32_ll_1000", "kind": "world", "algo": "ll", "shape": "", "world": 8, "dtype": "float32", "elems": 1000,
         "heap": False},
        # an fp32 bucket of a sharded optimizer
        {"name": "halves4_f32_bucket", "kind": "halves", "shape": "4", "world": 4, "dtype": "float32", "elems": BUCKET // 4},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nway"] * 6 + ["scaled"] * 2 + ["host", "world", "world", "world", "halves"])
    if kind == "nway":
        n = rng.choice([2, 2, 3, 4, 4, 5, 6, 7, 8, 8, 12, 16])
        op = "band" if rng.random() < 0.15 else "sum"
        dtype = rng.choice(["int32", "int64", "uint8"] if op == "band" else
                           ["float32"] * 4 + ["bfloat16"] * 4 + ["float16"] * 2 + ["float64", "int8", "int16", "int32", "int64"])
        # up to the bytes of bench.py's widest reduction
        elems = _spread(rng, 1000, (9 * 4 * (64 << 20)) // ((n + 1) * SIZE[dtype]) // 2)
        return {"kind": kind, "dtype": dtype, "op": op, "n": n, "elems": elems, "offset": rng.choice([0, 0, 0, 1, 4]),
                "out": rng.random() < 0.6}
    if kind == "scaled":
        return {"kind": kind, "in": rng.choice(["float32", "bfloat16"]), "to": rng.choice(["float32", "bfloat16"]),
                "n": rng.choice([2, 3, 4, 7, 8, 16]), "elems": _spread(rng, 1000, 16 << 20), "offset": rng.choice([0, 0, 0, 1])}
    if kind == "host":
        n = rng.choice([2, 3, 4, 8])
        return {"kind": kind, "dtype": rng.choice(["float32", "float32", "bfloat16", "int32"]), "n": n,
                "fanins": rng.choice([str(n), "2," + str(n)]), "elems": _spread(rng, 1000, 1 << 20)}
    if kind == "halves":
        world, shape = rng.choice([(2, "2"), (4, "4"), (4, "2*2"), (7, "2*3+1"), (8, "8"), (8, "2*4")])
        return {"kind": kind, "shape": shape, "world": world, "dtype": rng.choice(["float32", "bfloat16"]),
                "elems": _spread(rng, 4000, 8 << 20)}
    algo = rng.choice(["staged", "staged", "oneshot", "ll", "push"])
    world, shape = rng.choice([(2, "2"), (3, "3"), (4, "4"), (4, "2*2"), (5, "2*2+1"), (7, "2*3+1"), (8, "8"), (8, "2*4"),
                               (8, "2*2*2"), (8, "ring8")])
    dtype = rng.choice(["float32", "bfloat16", "float16"])
    if algo == "ll":     # a tree of tagged words, or the flat exchange
        return {"kind": kind, "algo": algo, "shape": rng.choice(["", shape]), "world": world, "dtype": dtype,
                "elems": _spread(rng, 100, (64 << 10) // SIZE[dtype]), "heap": False}
    if algo == "oneshot":
        return {"kind": kind, "algo": algo, "shape": str(world), "world": world, "dtype": dtype,
                "elems": _spread(rng, 1000, (1 << 20) // SIZE[dtype]), "heap": False}
    return {"kind": kind, "algo": algo, "shape": shape if algo == "staged" else str(world), "world": world, "dtype": dtype,
            "elems": _spread(rng, 4000, (32 << 20) // SIZE[dtype]), "heap": algo == "push" or rng.random() < 0.7}


def _vectors(n, elems, dtype, op, offset, seed):
    """n vectors of what the path meets: gradients (normal values), counters, masks.  ``offset``: elements between
    the start of an allocation and the vector in it."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    dt = getattr(torch, dtype)
    out = []
    for _ in range(n):
        if dtype in FLOATS:
            v = torch.randn(elems + offset, generator=g, device=DEVICE).to(dt)
        else:
            info = torch.iinfo(dt)
            lo, hi = (info.min, info.max) if op == "band" else (max(info.min, -1000), min(info.max, 1000))
            v = torch.randint(lo, hi, (elems + offset,), generator=g, device=DEVICE, dtype=dt)
        out.append(v[offset:])
    return out


def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind == "nway":
        s["in"] = _vectors(case["n"], case["elems"], case["dtype"], case["op"], case["offset"], seed)
        s["dst"] = torch.empty(case["elems"] + case["offset"], dtype=s["in"][0].dtype, device=DEVICE)[case["offset"]:] if case["out"] else None
    elif kind == "scaled":
        s["vec"] = _vectors(case["n"], case["elems"], case["in"], "sum", case["offset"], seed)
        s["dst"] = torch.empty(case["elems"] + case["offset"], dtype=getattr(torch, case["to"]), device=DEVICE)[case["offset"]:]
    elif kind == "host":
        s["fan"] = [int(x) for x in case["fanins"].split(",")]
        s["in"] = [torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v)
                   for v in _vectors(case["n"], case["elems"], case["dtype"], "sum", 0, seed)]
        s["dst"] = [torch.empty(case["elems"], dtype=s["in"][0].dtype, pin_memory=True) for _ in s["fan"]]
        s["pipe"] = HostReducePipeline(device=DEVICE, max_inputs=case["n"], max_outputs=len(s["fan"]))
    else:
        vec = _vectors(case["world"], case["elems"], case["dtype"], "sum", 0, seed)
        nbytes = case["elems"] * SIZE[case["dtype"]]
        heap = kind == "halves" or case["heap"]
        w = LocalWorld(case["world"], heap_bytes=nbytes + (1 << 20) if heap else 1 << 20,
                       staging_bytes=1 << 20 if heap else max(1 << 20, nbytes + (64 << 10)))
        s["comm"] = w
        if heap:   # averaged in place
            s["vec"] = [c.alloc(case["elems"], v.dtype) for c, v in zip(w.ranks, vec)]
            for t, v in zip(s["vec"], vec):
                t.copy_(v)
            s["dst"] = None
        else:
            s["vec"], s["dst"] = vec, [torch.empty_like(v) for v in vec]
    return s


def run(s):
    kind = s["kind"]
    if kind == "nway":
        return reduce_nway(s["in"], op=s["op"], out=s["dst"])
    if kind == "scaled":
        return reduce_nway_scaled(s["vec"], scale=1.0 / s["n"], out=s["dst"])
    if kind == "host":
        return s["pipe"].run(s["in"], s["fan"], s["dst"])
    if kind == "halves":
        s["comm"].reduce_scatter(s["vec"], op="avg", shape=s["shape"])
        return s["comm"].all_gather(s["vec"], shape=s["shape"])
    return s["comm"].all_reduce(s["vec"], op="avg", shape=s["shape"] or None, algo=s["algo"], outs=s["dst"])


def work(case):
    """Each input read once, each result written once; one addition per element folded in."""
    kind, e = case["kind"], case["elems"]
    if kind == "nway":
        return {"bytes": (case["n"] + 1) * e * SIZE[case["dtype"]], "flops": (case["n"] - 1) * e}
    if kind == "scaled":
        return {"bytes": case["n"] * e * SIZE[case["in"]] + e * SIZE[case["to"]], "flops": case["n"] * e}
    if kind == "host":
        fan = [int(x) for x in case["fanins"].split(",")]
        return {"bytes": (case["n"] + len(fan)) * e * SIZE[case["dtype"]], "flops": sum(f - 1 for f in fan) * e}
    return {"bytes": 2 * case["world"] * e * SIZE[case["dtype"]], "flops": case["world"] * e}


def tolerance(case):
    kind = case["kind"]
    dtype = case["to"] if kind == "scaled" else case["dtype"]
    if dtype not in FLOATS:
        return "exact"
    if dtype == "float64":
        return {"rel": 1e-14}
    if dtype == "float32":
        return {"rel": 1e-6}
    # one rounding of an fp32 sum; a plan of several levels rounds once per level
    levels = 1 if kind in ("nway", "scaled", "host") else 3
    return {"rel": levels * (4e-3 if dtype == "bfloat16" else 5e-4)}
