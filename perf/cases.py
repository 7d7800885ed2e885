"""The workloads this library's speed is measured on, as a program calls them on one GPU.

Two kinds of caller exist there. A job with a single rank uses its communicator as it would on
any number of GPUs. A program that holds all ranks of a small communicator on one device uses
the world entry points (`hxccl_b200.ops.world.World`), which run the same collective kernels for
every rank in one launch. The handles (communicator, worlds) are made once per process, as a
program does, and serve every buffer; nothing else is kept between calls.

Every result is defined bit for bit by the library's reduction orders, so results are compared
exactly.
"""
import math

import numpy as np
import torch

import hxccl_b200 as hx
from hxccl_b200.ops.world import World

DTYPES = {"fp32": (torch.float32, hx.FLOAT32), "bf16": (torch.bfloat16, hx.BFLOAT16), "fp16": (torch.float16, hx.FLOAT16),
          "fp8": (torch.float8_e4m3fn, hx.FLOAT8E4M3), "int32": (torch.int32, hx.INT32)}
SIZES = {"fp32": 4, "bf16": 2, "fp16": 2, "fp8": 1, "int32": 4}
OPS = {"sum": hx.SUM, "avg": hx.AVG, "max": hx.MAX}

# Parameters of one transformer block of the GPT-2 small in hxccl_b200/models (d_model 768): what
# a gradient bucket of the default 25 MB or one FSDP unit of that model holds.
BLOCK = 12 * 768 * 768 + 13 * 768
MIB = 1 << 20
# the most bytes a drawn case touches: as many as the largest listed one
MOST = 1 << 30

_handles: dict = {}


def _world(n: int) -> World:
    if n not in _handles:
        _handles[n] = World(n, window_mb=256, wait_ms=20000)
    return _handles[n]


def _communicator() -> hx.Communicator:
    if 1 not in _handles:
        torch.zeros(1, device="cuda")
        _handles[1] = hx.Communicator.init_rank(hx.get_unique_id(), 1, 0)
    return _handles[1]


def listed():
    return [
        # one rank: the out-of-place AllReduce that bench.py times by default
        {"name": "one_rank_sum", "kind": "allreduce", "ranks": 1, "dtype": "fp32", "op": "sum", "count": 64 * MIB, "in_place": False},
        # one rank: a data-parallel job tried on a single GPU averages its gradient buckets in place
        {"name": "one_rank_avg_bucket", "kind": "allreduce", "ranks": 1, "dtype": "fp32", "op": "avg", "count": BLOCK, "in_place": True},
        # a loss or a flag summed over all ranks: nothing but latency
        {"name": "scalar_pair", "kind": "allreduce", "ranks": 8, "dtype": "fp32", "op": "sum", "count": 2, "in_place": False},
        # a norm's or bias's gradient: below 64 KiB, so in the recursive-doubling order; an odd count
        {"name": "small_bf16_avg", "kind": "allreduce", "ranks": 8, "dtype": "bf16", "op": "avg", "count": 20487, "in_place": True},
        # an ordinary tensor of 16 MiB with a remainder in every block
        {"name": "medium_fp32_sum", "kind": "allreduce", "ranks": 4, "dtype": "fp32", "op": "sum", "count": 4 * MIB + 3, "in_place": False},
        # the largest message: 256 MiB per rank
        {"name": "large_fp32_sum", "kind": "allreduce", "ranks": 2, "dtype": "fp32", "op": "sum", "count": 64 * MIB, "in_place": False},
        # low-precision gradients: 16 MiB of e4m3, as in the low-precision benchmark
        {"name": "fp8_sum", "kind": "allreduce", "ranks": 8, "dtype": "fp8", "op": "sum", "count": 16 * MIB, "in_place": False},
        # gradient buckets after hxcclCommShrink took one of eight ranks out
        {"name": "seven_rank_bucket", "kind": "allreduce", "ranks": 7, "dtype": "fp32", "op": "avg", "count": BLOCK, "in_place": True},
        # the DDP hook with bf16 on the wire: cast, average and widen in one call
        {"name": "bf16_wire_bucket", "kind": "cast", "ranks": 8, "dtype": "bf16", "op": "avg", "count": BLOCK, "in_place": True},
        # a sharded step: gradients reduce-scattered, parameters all-gathered
        {"name": "sharded_step", "kind": "sharded", "ranks": 8, "dtype": "bf16", "op": "avg", "count": BLOCK // 8, "in_place": False},
        # uneven exchange: block sizes uniform in [0, 2 x mean] elements, so most blocks start off any alignment
        {"name": "uneven_exchange", "kind": "alltoallv", "ranks": 8, "dtype": "bf16", "op": "none", "count": MIB // 2, "in_place": False},
        # sequence parallelism: every rank sends its key/value block to the next one
        {"name": "ring_shift", "kind": "shift", "ranks": 4, "dtype": "bf16", "op": "none", "count": 16 * MIB, "in_place": False},
    ]


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "allreduce", "one", "cast", "sharded", "alltoallv", "shift"])
    ranks = rng.choice([2, 4, 8, 8]) if rng.random() < 0.75 else rng.choice([3, 5, 6, 7])
    dtype, op = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp16", "fp8", "int32"]), rng.choice(["sum", "sum", "avg", "max"])
    in_place = rng.random() < 0.4
    if kind == "one":
        kind, ranks = "allreduce", 1
    # smallest message in bytes, and the bytes touched per byte of it
    low, per = 8.0, 2.0 * ranks
    if kind == "cast":  # the call takes the ring order only: 64 KiB on the wire or more
        dtype, op, low, per = rng.choice(["bf16", "bf16", "fp16"]), rng.choice(["avg", "avg", "sum"]), 65536.0, 4.0 * ranks
    elif kind == "sharded":
        op, per = rng.choice(["sum", "avg"]), 2.0 * ranks * (ranks + 1)
    elif kind in ("alltoallv", "shift"):
        op, in_place = "none", False
        per = 2.0 * ranks * (ranks if kind == "alltoallv" else 1) * (2.0 if kind == "alltoallv" else 1.0)
    if kind == "sharded" or (op == "sum" and in_place):
        in_place = False
    # up to 256 MiB per rank, as the listed cases
    high = min(256.0 * MIB, MOST / per)
    count = max(1, int(math.exp(rng.uniform(math.log(low), math.log(high))) / SIZES[dtype]))
    if rng.random() < 0.5 and count > 64:
        count -= count % 64
    if kind == "cast":
        count = max(count, 65536 // SIZES[dtype])
    return {"kind": kind, "ranks": ranks, "dtype": dtype, "op": op, "count": count, "in_place": in_place}


def _values(count, dtype, gen):
    t = DTYPES[dtype][0]
    if dtype == "int32":
        return torch.randint(-1000, 1001, (count,), generator=gen, device="cuda", dtype=t)
    x = torch.randn(count, generator=gen, device="cuda", dtype=torch.float32)
    if dtype == "fp8":
        x.mul_(16)
    return x.to(t)


def prepare(case, seed):
    n, count, dtype = case["ranks"], case["count"], case["dtype"]
    t, es = DTYPES[dtype][0], SIZES[dtype]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = {"case": case, "dt": DTYPES[dtype][1], "op": OPS.get(case["op"]), "call": _communicator() if n == 1 else _world(n)}
    if case["kind"] == "alltoallv":
        rng = np.random.default_rng(7)  # the layout belongs to the case, the values to the seed
        nb = rng.integers(0, 2 * count + 1, (n, n)) * es  # nb[r][j]: bytes from rank r to rank j
        soff, roff = np.zeros_like(nb), np.zeros_like(nb)
        soff[:, 1:] = np.cumsum(nb, axis=1)[:, :-1]
        roff[:, 1:] = np.cumsum(nb.T, axis=1)[:, :-1]
        s["nbytes"], s["soff"], s["roff"] = nb.tolist(), soff.tolist(), roff.tolist()
        s["send"] = [_values(max(1, int(nb[r].sum()) // es), dtype, gen) for r in range(n)]
        s["recv"] = [torch.zeros(max(1, int(nb[:, r].sum()) // es), dtype=t, device="cuda") for r in range(n)]
        return s
    if case["kind"] == "sharded":
        s["send"] = [_values(count * n, dtype, gen) for _ in range(n)]    # gradients of the whole unit
        s["shard"] = [torch.zeros(count, dtype=t, device="cuda") for _ in range(n)]
        s["param"] = [_values(count, dtype, gen) for _ in range(n)]       # each rank's shard of the parameters
        s["recv"] = [torch.zeros(count * n, dtype=t, device="cuda") for _ in range(n)]
        return s
    s["send"] = [_values(count, "fp32" if case["kind"] == "cast" else dtype, gen) for _ in range(n)]
    s["recv"] = s["send"] if case["in_place"] else [torch.zeros_like(x) for x in s["send"]]
    if case["kind"] == "shift":
        s["transfers"] = [(r, (r + 1) % n, s["send"][r], count * es, s["recv"][(r + 1) % n], count * es) for r in range(n)]
    return s


def run(s):
    case, call = s["case"], s["call"]
    n, count = case["ranks"], case["count"]
    if case["kind"] == "alltoallv":
        call.all_to_allv(s["send"], s["recv"], s["nbytes"], s["soff"], s["roff"])
        return s["recv"]
    if case["kind"] == "shift":
        call.send_recv(s["transfers"])
        return s["recv"]
    if case["kind"] == "cast":
        call.all_reduce_cast(s["send"], s["recv"], count, s["dt"], op=s["op"])
        return s["recv"]
    if case["kind"] == "sharded":
        call.reduce_scatter(s["send"], s["shard"], count, s["dt"], op=s["op"])
        call.all_gather(s["param"], s["recv"], count * SIZES[case["dtype"]])
        return {"gradients": s["shard"], "parameters": s["recv"]}
    if n == 1:
        call.all_reduce(s["send"][0], s["recv"][0], op=s["op"])
    else:
        call.all_reduce(s["send"], s["recv"], count, s["dt"], op=s["op"])
    return s["recv"]


def work(case):
    n, nb = case["ranks"], case["count"] * SIZES[case["dtype"]]
    adds = (n - 1) * case["count"]
    if case["kind"] == "alltoallv":  # n * n blocks of nb bytes on average, read once and written once
        return {"bytes": 2 * n * n * nb, "flops": 0}
    if case["kind"] == "shift":
        return {"bytes": 2 * n * nb, "flops": 0}
    if case["kind"] == "cast":  # fp32 buffers
        return {"bytes": 2 * n * 4 * case["count"], "flops": adds}
    if case["kind"] == "sharded":  # n inputs of n blocks to n blocks; n blocks to n results of n blocks
        return {"bytes": 2 * (n * n + n) * nb, "flops": n * adds}
    return {"bytes": 2 * n * nb, "flops": adds}


def tolerance(case):
    return "exact"
