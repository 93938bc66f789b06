"""What is timed when this library's speed is measured: a list of cases over its public entry points.

Everything runs on one GPU.  A world of one is what a single-GPU (or per-rank) program has; a world of 2, 4
or 8 is the emulated one (`Communicator.virtual`): all ranks in one launch, one tensor per rank.

The kinds, and the ranges that the listed cases stand for and `draw` samples:

  allreduce        1 Ki - 16 Mi elements per rank, any count; the caller's own buffers (out of place) or buffers of
                   the symmetric heap (in place, filled by the program first)
  allgather        256 - 4 Mi elements per rank
  reduce_scatter   1 Ki - 16 Mi elements per rank
  allreduce_norm   all-reduce + residual + RMSNorm: 1 - 512 rows of 1024 - 8192
  linear           row-parallel linear + all-reduce, with or without residual + RMSNorm: 1 - 2048 rows, K 448 - 3584 per
                   rank, N 1024 - 8192 (up to 32 rows, as in decoding: the hidden sizes of a decoder, 4864 - 8192)
  gather_linear    all-gather + column-parallel linear: 1 - 8192 rows
  decode           one decode step of the Llama-shaped tensor-parallel decoder: batch 1 - 64, context 64 - 4096,
                   hidden 5120 - 8192

fp16 and bf16 throughout.  Shapes are the ones of the tests, of `bench.py`, `bench_fused_layer.py` and
`bench_decoder.py`: activations N(0, 1), weights N(0, 0.02), gamma around 1.
"""
from __future__ import annotations

import math

import torch

from gpu_ipc_example_b200 import Communicator, ops
from gpu_ipc_example_b200.models.llama import LlamaConfig, LlamaTP

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_EPS = 1e-5


def listed():
    return [
        # the smallest message of the sweep: launch and exchange latency
        dict(name="allreduce 2 KiB x8", kind="allreduce", world=8, n=1024, dtype="fp16", symmetric=False),
        # the activations of the reference's framework smoke test, [4, 1, 14336]
        dict(name="allreduce smoke x4", kind="allreduce", world=4, n=4 * 14336, dtype="fp16", symmetric=False),
        # the headline problem: 8 Mi elements per rank on symmetric buffers, in place
        dict(name="allreduce 16 MiB x8", kind="allreduce", world=8, n=8 << 20, dtype="fp16", symmetric=True),
        # an odd count in the caller's own buffers: gradients that nobody padded
        dict(name="allreduce odd x4", kind="allreduce", world=4, n=12345677, dtype="bf16", symmetric=False),
        # sharded activations or parameters put back together
        dict(name="allgather 1 MiB x8", kind="allgather", world=8, n=512 << 10, dtype="fp16", symmetric=False),
        # sharded gradients
        dict(name="reduce_scatter 16 MiB x8", kind="reduce_scatter", world=8, n=8 << 20, dtype="bf16", symmetric=False),
        # decode: the second half of a tensor-parallel block, 16 sequences
        dict(name="allreduce_norm 16 x8", kind="allreduce_norm", world=8, rows=16, hidden=8192, dtype="fp16"),
        # decode: the down-projection shard of a 70B-shaped layer at TP = 8, on the rank's own GPU
        dict(name="linear 16 x1", kind="linear", world=1, rows=16, k=3584, n=8192, dtype="fp16", norm=True),
        # prefill of the same layer
        dict(name="linear 2048 x1", kind="linear", world=1, rows=2048, k=3584, n=8192, dtype="fp16", norm=True),
        # a ragged prompt on two ranks, no norm behind it
        dict(name="linear 300 x2", kind="linear", world=2, rows=300, k=1792, n=8192, dtype="bf16", norm=False),
        # prefill of the gate/up projection on row-sharded activations
        dict(name="gather_linear 4096 x2", kind="gather_linear", world=2, rows=4096, k=8192, n=7168, dtype="fp16"),
        # four layers of the 70B-shaped decoder with the per-rank shapes of TP = 8: batch 32 at 2048 tokens
        dict(name="decode 32 x1", kind="decode", world=1, batch=32, ctx=2048, layers=4, hidden=8192, heads=8, kv_heads=1,
             ffn=3584, vocab=16032, dtype="fp16", fusion="gemm"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "allgather", "reduce_scatter", "allreduce_norm", "linear", "linear",
                       "gather_linear", "decode"])
    dtype = rng.choice(["fp16", "bf16"])
    world = rng.choice([2, 4, 8])
    if kind == "allreduce":
        return dict(kind=kind, world=world, n=_log(rng, 1 << 10, (128 << 20) // world // 2), dtype=dtype,
                    symmetric=rng.random() < 0.3)
    if kind == "allgather":
        return dict(kind=kind, world=world, n=2 * _log(rng, 128, (4 << 20) // world), dtype=dtype, symmetric=rng.random() < 0.3)
    if kind == "reduce_scatter":
        return dict(kind=kind, world=world, n=world * _log(rng, (1 << 10) // world, (64 << 20) // world // world), dtype=dtype,
                    symmetric=rng.random() < 0.3)
    if kind == "allreduce_norm":
        return dict(kind=kind, world=world, rows=_log(rng, 1, 512), hidden=8 * _log(rng, 128, 1024), dtype=dtype)
    if kind == "linear":
        world = rng.choice([1, 1, 2, 8])
        rows = _log(rng, 1, 2048 // world)
        return dict(kind=kind, world=world, rows=rows, k=8 * rng.randint(56, 448), n=64 * rng.randint(76 if rows <= 32 else 16, 128),
                    dtype=dtype, norm=rng.random() < 0.7)
    if kind == "gather_linear":
        world = rng.choice([1, 2, 4])
        return dict(kind=kind, world=world, rows=world * _log(rng, 1, 8192 // world // world), k=8 * rng.randint(64, 1024),
                    n=64 * rng.randint(4, 112), dtype=dtype)
    world = rng.choice([1, 1, 2])
    kv = rng.choice([1, 2, 4])
    return dict(kind="decode", world=world, batch=_log(rng, 1, 64), ctx=_log(rng, 64, 4096), layers=2, hidden=1024 * rng.randint(5, 8),
                heads=world * kv * rng.choice([1, 2, 4, 8 // kv]), kv_heads=world * kv, ffn=world * 128 * rng.randint(4, 28),
                vocab=16032, dtype=dtype, fusion=rng.choice(["gemm", "allreduce"]))


# ---------------------------------------------------------------------------------------------- preparation
_comms = {}


def _comm(case):
    """The communicator of a program that does this work: created once and kept."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _comms:
        w = case["world"]
        kind = case["kind"]
        if kind in ("allreduce", "reduce_scatter"):
            room = 4 * case["n"] * 2
        elif kind == "allgather":
            room = 4 * case["n"] * 2 * w
        elif kind == "allreduce_norm":
            room = 4 * case["rows"] * case["hidden"] * 2
        elif kind == "linear":
            room = 12 * max(case["rows"], 32) * case["n"] * 2
        elif kind == "gather_linear":
            room = 6 * case["rows"] * case["k"] * 2
        else:
            room = 64 * max(case["batch"], 32) * case["hidden"] * 2
        _comms[key] = (Communicator.virtual(w, 0, staging_bytes=room + (64 << 20)), {})
    return _comms[key]


def _symmetric(case, n):
    """One buffer per rank in the symmetric heap; allocated once, as the heap is."""
    comm, kept = _comm(case)
    if n not in kept:
        kept[n] = comm.empty([n], _DTYPES[case["dtype"]])
    return kept[n]


def prepare(case, seed):
    kind, w, dt = case["kind"], case["world"], _DTYPES[case["dtype"]]
    comm, _ = _comm(case)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dt)

    s = dict(case=case, comm=comm)
    if kind == "allreduce":
        s["x"] = [rnd(case["n"]) for _ in range(w)]
        s["out"] = _symmetric(case, case["n"]) if case["symmetric"] else [torch.empty_like(t) for t in s["x"]]
    elif kind == "allgather":
        s["x"] = [rnd(case["n"]) for _ in range(w)]
        s["out"] = _symmetric(case, w * case["n"]) if case["symmetric"] else [torch.empty(w * case["n"], device="cuda", dtype=dt) for _ in range(w)]
    elif kind == "reduce_scatter":
        s["x"] = [rnd(case["n"]) for _ in range(w)]
        if case["symmetric"]:
            s["buf"] = _symmetric(case, case["n"])
        s["out"] = [torch.empty(case["n"] // w, device="cuda", dtype=dt) for _ in range(w)]
    elif kind == "allreduce_norm":
        r, h = case["rows"], case["hidden"]
        s["x"] = [rnd(r, h) for _ in range(w)]
        s["res"] = [rnd(r, h)] * w
        s["gamma"] = [1 + rnd(h, scale=0.1)] * w
    elif kind == "linear":
        m, k, n = case["rows"], case["k"], case["n"]
        s["x"] = [rnd(m, k) for _ in range(w)]
        s["w"] = [rnd(n, k, scale=0.02) for _ in range(w)]
        s["res"] = [rnd(m, n)] * w
        s["gamma"] = [1 + rnd(n, scale=0.1)] * w
    elif kind == "gather_linear":
        m, k, n = case["rows"], case["k"], case["n"]
        s["x"] = [rnd(m // w, k) for _ in range(w)]
        s["w"] = [rnd(n, k, scale=0.02) for _ in range(w)]
    else:
        cfg = LlamaConfig(layers=case["layers"], hidden=case["hidden"], n_heads=case["heads"], n_kv_heads=case["kv_heads"],
                          ffn=case["ffn"], vocab=case["vocab"], dtype=dt)
        m = LlamaTP(cfg, comm, batch=case["batch"], max_ctx=case["ctx"], fusion=case["fusion"], seed=seed)
        for caches in (m.kcache, m.vcache):  # the tokens before this one
            for layer in (c for rank in caches for c in rank):
                layer.normal_(generator=g)
        s["model"] = m
        s["tokens"] = torch.randint(0, cfg.vocab, (case["batch"],), device="cuda", generator=g)
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    case, comm = s["case"], s["comm"]
    kind = case["kind"]
    if kind == "allreduce":
        if case["symmetric"]:
            for o, x in zip(s["out"], s["x"]):  # what produces the values writes them into the symmetric buffers
                o.copy_(x)
            return ops.all_reduce(s["out"], comm=comm)
        return comm.all_reduce(s["x"], s["out"])
    if kind == "allgather":
        return ops.all_gather_into_tensor(s["out"], s["x"], comm=comm)
    if kind == "reduce_scatter":
        if case["symmetric"]:
            for o, x in zip(s["buf"], s["x"]):
                o.copy_(x)
            return ops.reduce_scatter_tensor(s["out"], s["buf"], comm=comm)
        return ops.reduce_scatter_tensor(s["out"], s["x"], comm=comm)
    if kind == "allreduce_norm":
        return comm.allreduce_residual_rmsnorm(s["x"], s["res"], s["gamma"], _EPS)
    if kind == "linear":
        if case["norm"]:
            return comm.linear_allreduce(s["x"], s["w"], s["res"], s["gamma"], _EPS)
        return comm.linear_allreduce(s["x"], s["w"])
    if kind == "gather_linear":
        return comm.allgather_linear(s["x"], s["w"])
    m = s["model"]
    m.pos = case["ctx"] - 1  # the newest position of a full cache
    m.decode(s["tokens"])
    # The hidden states that the head's logits are a product of, and the caches with the new position in them.  The
    # greedy ids are left out: with random weights two logits of a row are often closer than the last bit.
    return m.last_hidden, m.kcache, m.vcache


# ---------------------------------------------------------------------------------------------- what it costs at least
def work(case):
    w, kind = case["world"], case["kind"]
    if kind == "allreduce":
        b = w * case["n"] * 2
        return {"bytes": 2 * b + (2 * b if case["symmetric"] else 0), "flops": w * case["n"]}
    if kind == "allgather":
        return {"bytes": w * case["n"] * 2 * (1 + w), "flops": 0}
    if kind == "reduce_scatter":
        b = w * case["n"] * 2
        return {"bytes": b + b // w + (2 * b if case["symmetric"] else 0), "flops": w * case["n"]}
    if kind == "allreduce_norm":
        b = case["rows"] * case["hidden"] * 2
        return {"bytes": w * 3 * b + b, "flops": w * case["rows"] * case["hidden"] * 6}
    if kind == "linear":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * (w * (m * k + n * k) + (w * 2 * m * n + m * n if case["norm"] else w * m * n)), "flops": 2 * w * m * n * k}
    if kind == "gather_linear":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * (m * k + w * (n * k + m * n)), "flops": 2 * w * m * n * k}
    h, hq, hkv, f, b = case["hidden"], case["heads"], case["kv_heads"], case["ffn"], case["batch"]
    weights = case["layers"] * ((hq + 2 * hkv) * 128 * h + h * hq * 128 + 3 * f * h) + case["vocab"] * h
    cache = case["layers"] * 2 * b * hkv * case["ctx"] * 128
    return {"bytes": 2 * (weights + cache), "flops": 2 * b * weights + 4 * case["layers"] * b * hq * case["ctx"] * 128}


def tolerance(case):
    if case["kind"] == "allgather":
        return "exact"
    half = case["dtype"] == "fp16"
    if case["kind"] == "decode":
        return {"rel": 8e-3 if half else 3e-2}
    if case["kind"] in ("linear", "allreduce_norm"):
        return {"rel": 1.5e-3 if half else 1e-2}
    return {"rel": 1e-3 if half else 7e-3}
