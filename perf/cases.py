"""Performance cases of the library: what its users have it do on one GPU, through the public entry points.

Three groups.  (1) Collectives as hccl_test issues them: `Communicator.all_reduce` and its siblings, algorithm left to the
selector, on a one-rank communicator and on communicators that hold every rank of a job in one process (the form
`hccl_test --local` uses where one GPU is all there is).  (2) The tensor-parallel MLP block on the fused GEMM kernels, at the
Llama-3-70B shape of the benchmark: prefill, a decode-sized batch, and split over four ranks.  (3) The expert-parallel
exchange of a mixture-of-experts layer (dispatch, then gate-weighted combine), for prefill and for a decode batch.

listed() names the cases, draw() makes more of the same ranges.  Communicators and MoE exchanges are kept from state to
state, as a program keeps them from step to step; inputs, outputs and weights belong to a state.
"""
import math
import os

# a wait that starves ends after half a minute instead of half an hour
os.environ.setdefault("HCCL_EXEC_TIMEOUT_MS", "30000")

import numpy as np
import torch

import cann_hccl_b200 as H
from cann_hccl_b200 import _lib as L
from cann_hccl_b200.models.tp_mlp import TensorParallelMLP
from cann_hccl_b200.parallel import moe

OPS = {"sum": L.SUM, "max": L.MAX}
ITEM = {"float32": 4, "bfloat16": 2, "float16": 2, "int32": 4}


def listed():
    return [
        # smallest message of the hccl_test sweep: launch and latency decide
        {"name": "allreduce_8KiB_8ranks", "kind": "allreduce", "ranks": 8, "count": 2048, "dtype": "float32", "op": "sum"},
        # a middle message of the max / bf16 half of the sweep; the count is odd, so that slices do not end on vectors
        {"name": "allreduce_1MB_bf16_max_4ranks", "kind": "allreduce", "ranks": 4, "count": 500003, "dtype": "bfloat16", "op": "max"},
        # largest message of the hccl_test sweep: a gradient bucket
        {"name": "allreduce_64MiB_8ranks", "kind": "allreduce", "ranks": 8, "count": 16 << 20, "dtype": "float32", "op": "sum"},
        # the headline benchmark on one GPU: a job that happens to run on a single rank still calls AllReduce
        {"name": "allreduce_64MiB_1rank", "kind": "allreduce", "ranks": 1, "count": 16 << 20, "dtype": "float32", "op": "sum"},
        # sharded data parallelism: gradients reduced to their owner (count is what one rank receives) ...
        {"name": "reduce_scatter_4MiB_bf16_8ranks", "kind": "reduce_scatter", "ranks": 8, "count": 2 << 20, "dtype": "bfloat16", "op": "sum"},
        # ... and parameters gathered back (count is what one rank gives), here with blocks that are not multiples of 16 bytes
        {"name": "allgather_1MiB_4ranks", "kind": "allgather", "ranks": 4, "count": 262147, "dtype": "float32"},
        # token exchange with an uneven count matrix, 1024 rows of 7168 from every rank
        {"name": "alltoallv_1024rows_8ranks", "kind": "alltoallv", "ranks": 8, "rows": 1024, "width": 7168, "matrix": 7, "dtype": "bfloat16"},
        # Llama-3-70B MLP, prefill of 8192 tokens: the benchmark's shape on one GPU
        {"name": "mlp_prefill_8192", "kind": "mlp", "ranks": 1, "tokens": 8192, "hidden": 8192, "ffn": 28672, "activation": "silu"},
        # the same block on a decode batch: one row block, the weights dominate
        {"name": "mlp_decode_128", "kind": "mlp", "ranks": 1, "tokens": 128, "hidden": 8192, "ffn": 28672, "activation": "silu"},
        # tensor parallel over four ranks (all in this process), a medium batch
        {"name": "mlp_tp4_2048", "kind": "mlp", "ranks": 4, "tokens": 2048, "hidden": 8192, "ffn": 28672, "activation": "silu"},
        # MoE exchange of the benchmark config on one GPU: 8192 tokens, 256 experts, top 8
        {"name": "moe_prefill_8192", "kind": "moe", "ranks": 1, "tokens": 8192, "hidden": 7168, "experts": 256, "topk": 8, "variant": "mesh"},
        # the same layer on a decode batch over four ranks
        {"name": "moe_decode_128_4ranks", "kind": "moe", "ranks": 4, "tokens": 128, "hidden": 7168, "experts": 256, "topk": 8, "variant": "mesh"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "reduce_scatter", "allgather", "alltoallv", "mlp", "mlp", "moe"])
    if kind in ("allreduce", "reduce_scatter", "allgather"):
        p = rng.choice([1, 2, 3, 4, 8] if kind == "allreduce" else [2, 3, 4, 8])
        dtype = rng.choice(["float32", "bfloat16", "float16", "int32"])
        # 8 KiB to 64 MiB a rank; ReduceScatter and AllGather count one rank's block of that
        nbytes = _log(rng, 8 << 10, 64 << 20) if kind == "allreduce" else _log(rng, 2 << 10, (64 << 20) // p)
        count = max(1, nbytes // ITEM[dtype])
        if rng.random() < 0.5:  # half of them whole numbers of vectors, as buckets are; half any number
            count = max(16, count // 16 * 16)
        case = {"kind": kind, "ranks": p, "count": count, "dtype": dtype}
        if kind != "allgather":
            case["op"] = rng.choice(["sum", "sum", "max"])
        return case
    if kind == "alltoallv":
        p = rng.choice([2, 3, 4, 8])
        width = rng.choice([7168, 4096, 2048, rng.randint(100, 5000)])
        rows = _log(rng, 8, min(4096, (1024 * 7168 * 8) // (width * p)))
        return {"kind": kind, "ranks": p, "rows": rows, "width": width, "matrix": rng.randint(0, 999), "dtype": rng.choice(["bfloat16", "float32"])}
    if kind == "mlp":
        p = rng.choice([1, 1, 2, 4])
        while True:
            tokens = 128 * p * max(1, int(round(_log(rng, 128, 8192) / (128 * p))))
            hidden, ffn = 256 * rng.randint(4, 32), 256 * p * rng.randint(max(1, 16 // p), 112 // p)
            if tokens <= 8192 and tokens * hidden * ffn >= 128 * 2048 * 8192:
                break
        return {"kind": kind, "ranks": p, "tokens": tokens, "hidden": hidden, "ffn": ffn, "activation": rng.choice(["silu", "silu", "gelu", "none"])}
    p = rng.choice([1, 2, 4, 8])
    return {"kind": "moe", "ranks": p, "tokens": _log(rng, 64, 8192 // p), "hidden": 256 * rng.randint(4, 28), "experts": rng.choice([64, 128, 256]),
            "topk": rng.choice([2, 4, 8]), "variant": rng.choice(["mesh", "mesh", "pairwise"])}


# ---------------------------------------------------------------------------------------------------------- state
_comms = {}
_exchange = {}


def _comm(p):
    """The job's communicator: one rank per process on a single GPU, or all p ranks of the job in this process."""
    if p not in _comms:
        if p == 1:
            _comms[p] = H.Communicator.init_root(1, H.Communicator.get_root_info(), 0, device=True)
        else:
            _comms[p] = H.Communicator.init_local(p, device=True, device_id=torch.cuda.current_device())
    return _comms[p]


def _moe_exchange(case):
    """The layer's exchange buffers: a model makes them once per shape.  One shape at a time is kept here."""
    key = (case["ranks"], case["tokens"], case["hidden"], case["experts"], case["topk"])
    if key not in _exchange:
        torch.cuda.synchronize()
        for ex in _exchange.values():
            ex.close()
        _exchange.clear()
        _exchange[key] = moe.MoEExchange(_comm(case["ranks"]), case["tokens"], case["hidden"], case["experts"], case["topk"])
    return _exchange[key]


def _rand(n, dtype, gen):
    """What hccl_test fills its buffers with: uniform [-1, 1), or small integers."""
    dt = getattr(torch, dtype)
    if not dt.is_floating_point:
        return torch.randint(-1000, 1000, (n,), device="cuda", dtype=dt, generator=gen)
    return torch.empty(n, device="cuda", dtype=torch.float32).uniform_(-1, 1, generator=gen).to(dt)


def _matrix(case):
    """Rows that rank i sends to rank j: every rank spreads its rows over the ranks by a popularity that is the case's own."""
    r = np.random.RandomState(case["matrix"])
    p = case["ranks"]
    pop = r.dirichlet(np.full(p, 4.0))
    return np.stack([r.multinomial(case["rows"], pop) for _ in range(p)]).astype(np.uint64)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, p = case["kind"], case["ranks"]
    comm = _comm(p)
    s = {"kind": kind, "comm": comm}
    if kind in ("allreduce", "reduce_scatter", "allgather"):
        n = case["count"]
        n_in, n_out = n * (p if kind == "reduce_scatter" else 1), n * (p if kind == "allgather" else 1)
        s["send"] = [_rand(n_in, case["dtype"], gen) for _ in range(p)]
        s["recv"] = [torch.zeros(n_out, device="cuda", dtype=x.dtype) for x in s["send"]]
        s["op"] = OPS[case.get("op", "sum")]
    elif kind == "alltoallv":
        m = _matrix(case) * np.uint64(case["width"])
        before = lambda c: np.concatenate([np.zeros((p, 1), np.uint64), np.cumsum(c, axis=1)[:, :-1]], axis=1).astype(np.uint64)
        sc, rc = np.ascontiguousarray(m), np.ascontiguousarray(m.T)
        s["counts"] = (sc, before(sc), rc, before(rc))
        s["send"] = [_rand(int(sc[r].sum()), case["dtype"], gen) for r in range(p)]
        s["recv"] = [torch.zeros(int(rc[r].sum()), device="cuda", dtype=s["send"][0].dtype) for r in range(p)]
    elif kind == "mlp":
        s["mlp"] = TensorParallelMLP(comm, case["hidden"], case["ffn"], seed=seed, activation=case["activation"])
        s["x"] = [torch.randn(case["tokens"] // p, case["hidden"], device="cuda", generator=gen).to(torch.bfloat16) for _ in range(p)]
    else:
        s["ex"], s["variant"] = _moe_exchange(case), case["variant"]
        s["x"] = [torch.randn(case["tokens"], case["hidden"], device="cuda", generator=gen).to(torch.bfloat16) for _ in range(p)]
        routed = [moe.route(case["tokens"], case["experts"], case["topk"], seed, r) for r in range(p)]
        s["idx"], s["gates"] = [i for i, _ in routed], [g for _, g in routed]
        s["out"] = [torch.empty_like(x) for x in s["x"]]
    if p == 1:  # a rank that is alone passes plain tensors, not lists with one entry per rank
        for k in ("send", "recv", "x", "idx", "gates", "out"):
            if k in s:
                s[k] = s[k][0]
    return s


def run(s):
    comm, kind = s["comm"], s["kind"]
    if kind == "allreduce":
        comm.all_reduce(s["send"], s["recv"], op=s["op"])
        return s["recv"]
    if kind == "reduce_scatter":
        comm.reduce_scatter(s["send"], s["recv"], op=s["op"])
        return s["recv"]
    if kind == "allgather":
        comm.all_gather(s["send"], s["recv"])
        return s["recv"]
    if kind == "alltoallv":
        sc, sd, rc, rd = s["counts"]
        comm.all_to_all_v(s["send"], sc, sd, s["recv"], rc, rd)
        return s["recv"]
    if kind == "mlp":
        return s["mlp"].forward(s["x"])
    # dispatch to the experts, combine what they return; the experts' own work is not this library's and is left out, so
    # that the combine reads the dispatched rows.  Row order inside an expert's group is free, hence not an output.
    ex = s["ex"]
    _, offsets, rows = ex.dispatch(s["x"], s["idx"], variant=s["variant"])
    out = ex.combine(s["gates"], variant=s["variant"], source="recv", out=s["out"])
    return out, offsets, rows


def work(case):
    kind, p = case["kind"], case["ranks"]
    if kind in ("allreduce", "reduce_scatter", "allgather"):
        block = case["count"] * ITEM[case["dtype"]]
        blocks = {"allreduce": 2 * p, "reduce_scatter": p * p + p, "allgather": p + p * p}[kind]
        adds = {"allreduce": p - 1, "reduce_scatter": p * (p - 1), "allgather": 0}[kind]  # every result once
        return {"bytes": block * blocks, "flops": adds * case["count"]}
    if kind == "alltoallv":
        return {"bytes": 2 * p * case["rows"] * case["width"] * ITEM[case["dtype"]], "flops": 0}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * (2 * t * h + 2 * h * f), "flops": 4 * t * h * f}
    # rows read, written to their experts, read back from the experts' output, and written combined
    t, h, k = p * case["tokens"], case["hidden"], case["topk"]
    return {"bytes": 2 * h * t * (2 + 2 * k) + 8 * t * k, "flops": 2 * t * k * h}


def tolerance(case):
    if case["kind"] in ("mlp", "moe"):
        return {"rel": 1e-2}  # bf16 results of fp32 sums
    if case.get("op") != "sum" or case["ranks"] == 1 or case["dtype"] == "int32":
        return "exact"
    return {"rel": 1e-5 if case["dtype"] == "float32" else 1e-2}
