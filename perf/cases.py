"""What this library is timed on: AllReduce and the casts around it, on one GPU, through the public entry points.

Four entry points, each with what a program keeps between calls in its state:

``comm``    ``ops.LocalComm(n, emulate=True).run(program, tensors)``: the compiled schedule of all n ranks in one
            launch on one device, in place, with the mean fused (the gradient average of data-parallel training).
``staged``  the same with ``user_tensors``: gradient buckets that peers cannot reach, copied in, reduced on the wire
            type and copied out by the same kernel.
``c10d``    ``torch.distributed`` with backend ``stragglar`` on a group of one rank: ``dist.all_reduce`` of a tensor of
            the symmetric heap (what ``bench.py`` times on one GPU) or of an ordinary tensor, and
            ``parallel.all_reduce_ex`` with another type on the wire.
``cast``    ``ops.scale_cast``: gradients to and from the wire type with the division by the world size fused.

Sizes are those of the repository's own programs: the 4 KiB to 1 GiB of ``bench/sweep.sh`` and
``bench/backend_allreduce.py``, DDP's 25 MiB bucket, the 1 GiB of ``bench.py``, and the ragged element counts of
``tests/``.  A collective is run on the tensors that the last one left, as a training step does; with the mean fused
the values keep their magnitude.
"""
import math
import os

import torch

from stragglar_b200 import ops
from stragglar_b200.compiler import compile_program

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
MIB = 1 << 20
BENCH_COUNT = math.ceil((1 << 30) / (1024 * 7)) * 1024 * 7 // 4      # bench.py's default buffer, in fp32 elements


def _comm(name, alg, n, count, dtype, path):
    return {"name": name, "entry": "comm", "alg": alg, "n": n, "count": count, "dtype": dtype, "path": path}


def _staged(name, alg, n, count, dtype, wire, path):
    return {"name": name, "entry": "staged", "alg": alg, "n": n, "count": count, "dtype": dtype, "wire": wire, "path": path}


def listed():
    return [
        # a norm, a loss or a handful of control values: pure latency
        _comm("rsag_8r_4KiB_fp32", "rsag", 8, 1024, "fp32", "tma"),
        # a small layer's gradients, between latency and bandwidth
        _comm("a2a_8r_1MiB_bf16", "stragglar_a2a", 8, 512 * 1024, "bf16", "tma"),
        # the synthesized schedule at DDP's bucket size, in the symmetric heap
        _comm("stragglar_8r_25MiB_fp32", "stragglar", 8, 25 * MIB // 4, "fp32", "tma"),
        # the same bucket as DDP hands it over: an ordinary tensor
        _staged("stragglar_8r_bucket_fp32", "stragglar", 8, 25 * MIB // 4, "fp32", "fp32", "tma"),
        # bf16_fused_avg_hook's bucket: fp32 at the caller, bf16 on the wire, a ragged count
        _staged("rsag_8r_bucket_bf16_wire", "rsag", 8, 6_553_601, "fp32", "bf16", "tma"),
        # a flat gradient buffer, the size at which the rounds of the schedule are gated
        _comm("stragglar_8r_256MiB_fp32", "stragglar", 8, 64 * MIB, "fp32", "tma"),
        # a group that is no power of two, a count that is no multiple of anything, the communicator's default path
        _comm("stragglar_6r_ragged_fp32", "stragglar", 6, 3_000_017, "fp32", "simt"),
        # the baselines that the benchmark program offers beside the schedule
        _comm("ring_4r_40MB_fp32", "ring", 4, 10_000_019, "fp32", "simt"),
        _comm("rhd_8r_64MiB_fp16", "rhd", 8, 32 * MIB, "fp16", "simta"),
        # bench.py on one GPU: dist.all_reduce of 1 GiB in the symmetric heap
        {"name": "c10d_symmetric_1GiB_fp32", "entry": "c10d", "count": BENCH_COUNT, "dtype": "fp32", "wire": "fp32",
         "symmetric": True},
        # dist.all_reduce of an ordinary 64 KiB tensor: the host path of the backend and one staged kernel
        {"name": "c10d_ordinary_64KiB_fp32", "entry": "c10d", "count": 16 * 1024, "dtype": "fp32", "wire": "fp32",
         "symmetric": False},
        # gradients to the wire type before the two-phase collectives
        {"name": "cast_100MB_fp32_bf16", "entry": "cast", "count": 25_000_003, "dtype": "fp32", "wire": "bf16"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["comm", "comm", "comm", "comm", "staged", "staged", "c10d", "cast"])
    dtype = rng.choice(["fp32", "fp32", "bf16", "fp16"])
    esize = 4 if dtype == "fp32" else 2
    if entry == "cast":
        other = rng.choice([d for d in ("fp32", "bf16", "fp16") if d != dtype])
        return {"entry": "cast", "count": _log_uniform(rng, 1000, 64 * MIB), "dtype": dtype, "wire": other}
    if entry == "c10d":
        symmetric = rng.random() < 0.5
        wire = dtype if symmetric else rng.choice([dtype, "bf16"])
        return {"entry": "c10d", "count": _log_uniform(rng, 1024, 64 * MIB), "dtype": dtype, "wire": wire,
                "symmetric": symmetric}
    n = rng.choice([2, 4, 6, 8, 8])
    algs = ["stragglar", "stragglar_a2a", "ring", "rsag"]
    if n & (n - 1) == 0:
        algs.append("rhd")
    if entry == "comm" and n > 2:
        algs.append("direct")
    # 4 KiB to 64 MiB a rank (32 MiB of a caller's tensors): less than the largest listed case, whatever the algorithm
    count = _log_uniform(rng, 4096 // esize, (32 if entry == "staged" else 64) * MIB // esize)
    path = rng.choice(["tma", "tma", "simt", "simta"])
    if entry == "staged":
        return {"entry": "staged", "alg": rng.choice(algs), "n": n, "count": count, "dtype": dtype,
                "wire": rng.choice([dtype, "bf16"]), "path": path}
    return {"entry": "comm", "alg": rng.choice(algs), "n": n, "count": count, "dtype": dtype, "path": path}


_group = None
_comms = {}


def _communicator(n):
    """The communicator of n ranks that the program keeps: its collectives follow one another on its stream."""
    if n not in _comms:
        _comms[n] = ops.LocalComm(n, emulate=True)
    return _comms[n]


def _process_group():
    """The process group of the program: one rank, made once, with room for a few buffers of the largest case."""
    global _group
    if _group is None:
        import torch.distributed as dist
        import stragglar_b200.parallel as sp
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        sp.configure(arena_bytes=6 << 30, staging_bytes=256 << 20)
        dist.init_process_group("stragglar", store=dist.HashStore(), rank=0, world_size=1)
        _group = (dist, sp)
    return _group


def _gradients(count, dtype, seed, rank):
    """Gradients as a rank holds them: normal, with a standard deviation of 1e-2."""
    g = torch.Generator(device="cuda").manual_seed(seed * 64 + rank)
    return torch.empty(count, device="cuda").normal_(0.0, 1e-2, generator=g).to(DTYPES[dtype])


def prepare(case, seed):
    entry, count, dtype = case["entry"], case["count"], case["dtype"]
    if entry == "cast":
        return {"case": case, "src": _gradients(count, dtype, seed, 0),
                "dst": torch.empty(count, device="cuda", dtype=DTYPES[case["wire"]])}
    if entry == "c10d":
        dist, sp = _process_group()
        x = _gradients(count, dtype, seed, 0)
        if case["symmetric"]:
            s = sp.empty_symmetric(count, dtype=DTYPES[dtype], device="cuda")
            s.copy_(x)
            x = s
        return {"case": case, "x": x}
    n = case["n"]
    grads = [_gradients(count, dtype, seed, r) for r in range(n)]
    state = {"case": case, "comm": _communicator(n), "program": compile_program(case["alg"], n), "grads": grads}
    if entry == "staged":
        state["arena"] = [torch.zeros(count, device="cuda", dtype=DTYPES[case["wire"]]) for _ in range(n)]
    return state


def run(state):
    case = state["case"]
    if case["entry"] == "cast":
        ops.scale_cast(state["dst"], state["src"], 1.0 / 8)
        return state["dst"]
    if case["entry"] == "c10d":
        dist, sp = _group
        if case["wire"] == case["dtype"]:
            dist.all_reduce(state["x"], op=dist.ReduceOp.AVG)
        else:
            sp.all_reduce_ex(state["x"], average=True, comm_dtype=DTYPES[case["wire"]]).wait()
        return state["x"]
    n = case["n"]
    if case["entry"] == "staged":
        state["comm"].run(state["program"], state["arena"], path=case["path"], scale=1.0 / n, user_tensors=state["grads"])
    else:
        state["comm"].run(state["program"], state["grads"], path=case["path"], scale=1.0 / n)
    return state["grads"]


def _esize(dtype):
    return 4 if dtype == "fp32" else 2


def work(case):
    """Every rank's gradients read once and the mean written once to every rank."""
    count, es = case["count"], _esize(case["dtype"])
    if case["entry"] == "cast":
        return {"bytes": count * (es + _esize(case["wire"])), "flops": count}
    n = case.get("n", 1)
    return {"bytes": 2 * n * count * es, "flops": n * count}


def tolerance(case):
    """About four times what the tables show against sums in 64 bits of the same (wire-rounded) inputs: up to 6e-8 in
    fp32, 4.6e-4 in fp16 and, in bf16, 1.7e-3 to 2.4e-3 (3.7e-3 for the ring, which rounds at every rank)."""
    if case["entry"] in ("cast", "c10d"):      # one product and one rounding an element: nothing to choose
        return "exact"
    types = {case["dtype"], case.get("wire", case["dtype"])}
    if "bf16" in types:
        return {"rel": 1.0e-2}
    if "fp16" in types:
        return {"rel": 1.5e-3}
    return {"rel": 5e-7}


def exact(case, seed):
    """The scaled gradients (cast), the gradients themselves (a group of one rank) or their mean at every rank, in 64
    bits.  The wire's rounding is part of what a group of one rank returns; elsewhere it is the implementation's error."""
    count, dtype = case["count"], case["dtype"]
    if case["entry"] == "cast":
        return _gradients(count, dtype, seed, 0).double() * (1.0 / 8)
    if case["entry"] == "c10d":
        return _gradients(count, dtype, seed, 0).to(DTYPES[case["wire"]]).double()
    mean = torch.zeros(count, device="cuda", dtype=torch.float64)
    for r in range(case["n"]):
        mean += _gradients(count, dtype, seed, r).double()
    mean /= case["n"]
    return [mean] * case["n"]
