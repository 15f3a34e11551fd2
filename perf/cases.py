"""The calls whose speed this library answers for, on one GPU.

Six families, each through the entry point a program uses:

* ``group``   - ``EmuGroup.run``: the cross-rank kernels (low-latency, zero-copy, staged) over buffers of one device
* ``landing`` - ``reduce_landing``: folding landed chunks, from device memory or from pinned host memory
* ``dist``    - ``torch.distributed`` on the ``hylink`` backend with one rank
* ``zero``    - ``ShardedAdamW.step``: reduce-scatter, sharded AdamW, all-gather
* ``moe``     - ``ExpertParallelMLP``: routing, dispatch, experts, combine; forward and backward
* ``ddp``     - ``DDPTrainer.step``: the GPT-2 training step from a pinned host batch to the loss on the host
"""
import math

import torch
import torch.distributed as dist

from hylink_b200.models.gpt2 import GPT2, GPT2Config
from hylink_b200.ops import EmuGroup, reduce_landing
from hylink_b200.parallel.moe import ExpertParallelMLP
from hylink_b200.parallel.trainer import DDPTrainer, init_distributed
from hylink_b200.parallel.zero import ShardedAdamW

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
MIB = 1 << 20


def listed():
    return [
        # a small tensor-parallel activation or metric: latency, one launch
        group("allreduce_64k_8r", "all_reduce", 8, 32 << 10, "bf16"),
        # one 25 MB gradient bucket of the data-parallel trainer, in registered memory, averaged
        group("allreduce_bucket_4r", "all_reduce", 4, 25 * MIB // 2, "bf16", registered=True, op="avg"),
        # fp32 gradients in ordinary tensors, a count that is no multiple of anything
        group("allreduce_ragged_8r", "all_reduce", 8, 4 * MIB - 3, "fp32"),
        # sharded gradients: 64 MiB of fp32 per rank
        group("reducescatter_64m_4r", "reduce_scatter", 4, 4 * MIB, "fp32"),
        # sharded parameters: 16 MiB of bf16 from every rank
        group("allgather_64m_4r", "all_gather", 4, 8 * MIB, "bf16"),
        # expert-parallel dispatch: 8192 tokens of width 1024 per rank
        group("alltoall_16m_8r", "all_to_all", 8, MIB, "bf16"),
        # four landed 32 MiB contributions folded and averaged in one pass
        {"name": "landing_device_4x32m", "kind": "landing", "sources": 4, "count": 16 * MIB, "dtype": "bf16", "host": False,
         "accumulate": False, "scale": 0.25},
        # three peers' slices in pinned host memory folded into the local one; the last slice of a message is ragged
        {"name": "landing_host_3x4m", "kind": "landing", "sources": 3, "count": MIB - 5, "dtype": "fp32", "host": True,
         "accumulate": True, "scale": 1.0},
        # a reduce-scatter and an all-gather of a one-rank job
        {"name": "dist_pair_2m", "kind": "dist", "count": MIB, "dtype": "bf16"},
        # the optimizer step over a GPT-2-medium of bf16 weights with fp32 master copies
        {"name": "zero_step_medium", "kind": "zero", "layers": 24, "width": 1024, "vocab": 50257, "dtype": "bf16"},
        # a mixture-of-experts layer on 8192 tokens, capacity factor 1.25
        {"name": "moe_8192x1024", "kind": "moe", "tokens": 8192, "width": 1024, "hidden": 4096, "experts": 8, "capacity": 1280},
        # the benchmark's training step
        {"name": "ddp_gpt2_medium", "kind": "ddp", "model": "gpt2-medium", "batch": 8, "seq": 1024},
    ]


def group(name, coll, ranks, count, dtype, registered=False, op="sum", wire=""):
    """`count`: elements of the buffer (all-reduce, broadcast) or of one segment (the others)."""
    return {"name": name, "kind": "group", "coll": coll, "ranks": ranks, "count": count, "dtype": dtype, "registered": registered, "op": op,
            "wire": wire}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["group"] * 6 + ["landing"] * 2 + ["dist", "zero", "moe", "ddp"])
    if kind == "group":
        coll = rng.choice(["all_reduce"] * 3 + ["reduce_scatter", "all_gather", "all_to_all", "broadcast"])
        ranks = rng.choice([2, 4, 8])
        dtype = rng.choice(["bf16", "bf16", "fp32", "fp16"])
        registered = coll != "all_to_all" and rng.random() < 0.4
        segments = 1 if coll in ("all_reduce", "broadcast") else ranks
        count = _log(rng, 512, 256 * MIB // ranks // segments // SIZE[dtype])
        if registered or rng.random() < 0.5:  # whole 16-byte packets; else whatever came
            count = max(8, count // 8 * 8)
        wire = "bf16" if coll == "all_reduce" and dtype == "fp32" and not registered and rng.random() < 0.3 else ""
        c = group("", coll, ranks, count, dtype, registered, rng.choice(["sum", "avg"]) if "reduce" in coll else "sum", wire)
        del c["name"]
        return c
    if kind == "landing":
        host = rng.random() < 0.4
        return {"kind": kind, "sources": rng.randint(1, 7), "count": _log(rng, 1 << 10, (2 if host else 16) * MIB), "dtype": rng.choice(list(DTYPES)),
                "host": host, "accumulate": rng.random() < 0.5, "scale": rng.choice([1.0, 1.0, 0.5])}
    if kind == "dist":
        return {"kind": kind, "count": _log(rng, 1 << 10, 256 * MIB), "dtype": rng.choice(["bf16", "fp32"])}
    if kind == "zero":
        width = 64 * rng.randint(2, 16)
        return {"kind": kind, "layers": rng.randint(2, 24), "width": width, "vocab": rng.randint(1000, 50257), "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "moe":
        tokens, experts = _log(rng, 64, 8192), rng.choice([2, 4, 8])
        width = 64 * rng.randint(4, 16)
        return {"kind": kind, "tokens": tokens, "width": width, "hidden": 4 * width, "experts": experts, "capacity": max(1, int(1.25 * tokens / experts))}
    return {"kind": kind, "model": rng.choice(["tiny", "gpt2-small", "gpt2-medium"]), "batch": rng.randint(1, 8), "seq": rng.randint(16, 128) * rng.choice([1, 1, 8])}


def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def _one_rank_job():
    torch.cuda.set_device(0)
    if not dist.is_initialized():
        init_distributed("hylink")


def prepare(case, seed):
    return {"case": case, **{"group": _prepare_group, "landing": _prepare_landing, "dist": _prepare_dist, "zero": _prepare_zero,
                             "moe": _prepare_moe, "ddp": _prepare_ddp}[case["kind"]](case, seed)}


def run(state):
    return {"group": _run_group, "landing": _run_landing, "dist": _run_dist, "zero": _run_zero, "moe": _run_moe,
            "ddp": _run_ddp}[state["case"]["kind"]](state)


# ---------------------------------------------------------------- group
def _group_elements(c):
    """(elements of one rank's input, of one rank's output)"""
    n, k = c["ranks"], c["count"]
    return {"all_reduce": (k, k), "broadcast": (k, k), "reduce_scatter": (n * k, k), "all_gather": (k, n * k), "all_to_all": (n * k, n * k)}[c["coll"]]


def _prepare_group(c, seed):
    torch.cuda.set_device(0)
    g, gen, dt = EmuGroup(c["ranks"]), _gen(seed), DTYPES[c["dtype"]]
    n_in, n_out = _group_elements(c)
    if c["registered"]:
        ins, outs = g.alloc_registered(n_in, dt), g.alloc_registered(n_out, dt)
    else:
        ins, outs = ([torch.empty(k, dtype=dt, device="cuda") for _ in range(c["ranks"])] for k in (n_in, n_out))
    for t in ins:
        t.normal_(generator=gen)
    options = {"op": c["op"]}
    if c["coll"] in ("reduce_scatter", "all_to_all"):
        options["in_seg_stride"] = c["count"]
    if c["coll"] in ("all_gather", "all_to_all"):
        options["out_seg_stride"] = c["count"]
    if c["wire"]:
        options["wire_dtype"] = DTYPES[c["wire"]]
    return {"group": g, "ins": ins, "outs": outs, "options": options}


def _run_group(s):
    s["group"].run(s["case"]["coll"], s["ins"], s["outs"], s["case"]["count"], **s["options"])
    return s["outs"]


# ---------------------------------------------------------------- landing
def _prepare_landing(c, seed):
    torch.cuda.set_device(0)
    dt = DTYPES[c["dtype"]]
    gen = _gen(seed, "cpu" if c["host"] else "cuda")
    srcs = [torch.empty(c["count"], dtype=dt, pin_memory=True) if c["host"] else torch.empty(c["count"], dtype=dt, device="cuda")
            for _ in range(c["sources"])]
    for t in srcs:
        t.normal_(generator=gen)
    # an accumulating destination grows by the same contributions on every pass; 16-bit ones stop growing by themselves
    return {"srcs": srcs, "dst": torch.zeros(c["count"], dtype=dt, device="cuda")}


def _run_landing(s):
    c = s["case"]
    return reduce_landing(s["dst"], s["srcs"], scale=c["scale"], accumulate=c["accumulate"])


# ---------------------------------------------------------------- dist
def _prepare_dist(c, seed):
    _one_rank_job()
    dt = DTYPES[c["dtype"]]
    full = torch.empty(c["count"], dtype=dt, device="cuda").normal_(generator=_gen(seed))
    return {"full": full, "shard": torch.empty_like(full), "gathered": torch.empty_like(full)}


def _run_dist(s):
    dist.reduce_scatter_tensor(s["shard"], s["full"])
    dist.all_gather_into_tensor(s["gathered"], s["shard"])
    return s["shard"], s["gathered"]


# ---------------------------------------------------------------- zero
def _zero_parameters(c):
    """Shapes of a GPT-2 of these dimensions."""
    d = c["width"]
    block = [(d,), (d,), (3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (4 * d, d), (4 * d,), (d, 4 * d), (d,)]
    return [(c["vocab"], d), (1024, d), (d,), (d,)] + block * c["layers"]


def _zero_count(c):
    return sum(math.prod(s) for s in _zero_parameters(c))


def _prepare_zero(c, seed):
    _one_rank_job()
    gen, dt = _gen(seed), DTYPES[c["dtype"]]
    params = [torch.nn.Parameter(torch.empty(s, dtype=dt, device="cuda").normal_(std=0.02, generator=gen)) for s in _zero_parameters(c)]
    opt = ShardedAdamW(params, lr=3e-4, weight_decay=0.1)
    opt.flat_grad.normal_(std=1e-3, generator=gen)  # what a backward pass leaves there
    return {"opt": opt}


def _run_zero(s):
    o = s["opt"]
    o.step()
    return {"flat": o.flat, "m": o.m, "v": o.v, **({"master": o.master} if o.master is not None else {})}


# ---------------------------------------------------------------- moe
def _prepare_moe(c, seed):
    _one_rank_job()
    torch.manual_seed(seed)
    with torch.device("cuda"):
        layer = ExpertParallelMLP(c["width"], c["hidden"], experts_per_rank=c["experts"], capacity=c["capacity"]).to(torch.bfloat16)
    gen = _gen(seed)
    x = torch.empty(c["tokens"], c["width"], dtype=torch.bfloat16, device="cuda").normal_(generator=gen).requires_grad_(True)
    return {"layer": layer, "x": x, "dy": torch.empty_like(x).normal_(generator=gen)}


def _run_moe(s):
    layer, x = s["layer"], s["x"]
    layer.zero_grad(set_to_none=True)
    x.grad = None
    y = layer(x)
    y.backward(s["dy"])
    return {"y": y, "dx": x.grad, **{name: p.grad for name, p in layer.named_parameters()}}


# ---------------------------------------------------------------- ddp
def _prepare_ddp(c, seed):
    _one_rank_job()
    torch.manual_seed(seed)
    config = GPT2Config.by_name(c["model"])
    with torch.device("cuda"):
        model = GPT2(config)
    trainer = DDPTrainer(model, torch.device("cuda", 0))
    tokens = torch.randint(0, config.vocab_size, (c["batch"], min(c["seq"], config.n_ctx) + 1), generator=_gen(seed, "cpu")).pin_memory()
    return {"trainer": trainer, "tokens": tokens}


def _run_ddp(s):
    t = s["trainer"]
    loss = t.step(s["tokens"])
    params = list(t.model.parameters())
    # the weights and the gradients as one tensor each: there are hundreds of them
    return {"loss": loss, "weights": torch.cat([p.detach().reshape(-1) for p in params]), "gradients": torch.cat([p.grad.reshape(-1) for p in params])}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    if c["kind"] == "group":
        n_in, n_out = _group_elements(c)
        inputs = 1 if c["coll"] == "broadcast" else c["ranks"]
        adds = (c["ranks"] - 1) * c["count"] * (c["ranks"] if c["coll"] == "reduce_scatter" else 1)
        return {"bytes": (inputs * n_in + c["ranks"] * n_out) * SIZE[c["dtype"]], "flops": adds if "reduce" in c["coll"] else 0}
    if c["kind"] == "landing":
        operands = c["sources"] + c["accumulate"]
        return {"bytes": (operands + 1) * c["count"] * SIZE[c["dtype"]], "flops": (operands - 1 + (c["scale"] != 1.0)) * c["count"]}
    if c["kind"] == "dist":
        return {"bytes": 4 * c["count"] * SIZE[c["dtype"]], "flops": 0}
    if c["kind"] == "zero":
        # gradient in, weight out, both moments in and out; the fp32 master in and out, or the fp32 weight in
        n, es = _zero_count(c), SIZE[c["dtype"]]
        return {"bytes": n * (2 * es + 16 + (8 if es == 2 else 4)), "flops": 15 * n}
    if c["kind"] == "moe":
        rows = min(c["tokens"], c["experts"] * c["capacity"])
        weights = 2 * c["experts"] * c["width"] * c["hidden"] + c["experts"] * c["width"]
        # forward, and backward to the inputs and to the weights; x, dy, weights in, y, dx, weight gradients out
        return {"bytes": 2 * (4 * c["tokens"] * c["width"] + 2 * weights),
                "flops": 3 * 2 * (rows * 2 * c["width"] * c["hidden"] + c["tokens"] * c["width"] * c["experts"])}
    m = GPT2Config.by_name(c["model"])
    seq = min(c["seq"], m.n_ctx)
    tokens = c["batch"] * seq
    matrices = 12 * m.n_layer * m.d_model ** 2 + m.vocab_size * m.d_model
    params = matrices + m.n_ctx * m.d_model + m.n_layer * 13 * m.d_model + 2 * m.d_model
    # weights and both moments in and out, gradients out; all in bf16; causal attention is half a square
    return {"bytes": 14 * params + 8 * tokens, "flops": 6 * matrices * tokens + 6 * m.n_layer * tokens * seq * m.d_model}


def tolerance(case):
    c = case
    if c["kind"] == "dist" or c.get("coll") in ("all_gather", "all_to_all", "broadcast"):
        return "exact"
    if c["kind"] in ("group", "landing"):  # fp32 accumulation, one rounding
        return {"rel": 1e-6, "max": 1e-5} if c["dtype"] == "fp32" and not c.get("wire") else {"rel": 4e-3, "max": 1e-2}
    if c["kind"] == "zero":  # fp32 moments and master weights, rounded to the weights' type
        return {"rel": 1e-5, "max": 1e-4} if c["dtype"] == "fp32" else {"rel": 1e-3, "max": 1e-2}
    if c["kind"] == "moe":
        return {"rel": 1e-2}
    return {"rel": 2e-2, "max": 0.9}  # 24 bf16 layers forward and back; an Adam step takes the sign of the smallest gradients
