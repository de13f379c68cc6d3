"""The calls whose speed this repository watches: MoE FFN layers and dense FFN blocks on GGUF-quantised weights, through
the host wrappers of b200moe.ops, as a model's decode and prefill loops make them.

  listed()             the fixed cases
  draw(rng)            another case of the same ranges
  prepare(case, seed)  weights, handles and activations on the GPU, made from the seed
  run(state)           one call
  work(case)           the bytes and operations that the call cannot do without
  tolerance(case)      how far apart two correct implementations may be

Three kinds of call:
  ffn    MoeFfn: router, A8 activations, routed experts and combine in one call; with `shared` the shared expert (a Q8_0
         dense block) runs first and its output is folded in by the combine.
  layer  the operator chain of an engine that keeps its own router: RMSNorm + A8, router, routed layer with a bfloat16
         copy of the result.
  dense  A8 activations and a dense SwiGLU block.
Tensor types are ggml type ids: 7 Q5_1, 8 Q8_0, 12 Q4_K, 13 Q5_K.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("strix-halo-engine-lab_b200"))
import b200moe  # noqa: E402
from b200moe import ops  # noqa: E402

BLOCK = {7: (32, 24), 8: (32, 34), 12: (256, 144), 13: (256, 176)}  # values and bytes of a block
SHARED_TYPE = 8


def _ffn(name, rows, hidden, inter, experts, top_k, gate, down, bf16=False, zipf=False, groups=0, shared=False, kind="ffn"):
    return {"name": name, "kind": kind, "rows": rows, "hidden": hidden, "inter": inter, "experts": experts, "top_k": top_k, "gate": gate,
            "down": down, "bf16": bf16, "zipf": zipf, "groups": groups, "shared": shared}


def _dense(name, rows, hidden, inter, quant=12, bf16=False):
    return {"name": name, "kind": "dense", "rows": rows, "hidden": hidden, "inter": inter, "gate": quant, "down": quant, "bf16": bf16}


def listed():
    return [
        # one token through a small Q8_0 layer: single-stream decode, the least work a call can have
        _ffn("q8_0_decode_1", 1, 2048, 1024, 64, 4, 8, 8),
        # a prompt through the same layer
        _ffn("q8_0_prefill_512", 512, 2048, 1024, 64, 4, 8, 8, bf16=True),
        # single-stream decode and a batch of eight on the 128-expert Q4_K layer
        _ffn("q4_k_decode_1", 1, 2048, 768, 128, 8, 12, 12),
        _ffn("q4_k_decode_8", 8, 2048, 768, 128, 8, 12, 12),
        # a ragged serving batch: more rows than a decode batch, fewer than a prompt
        _ffn("q4_k_window_37", 37, 2048, 768, 128, 8, 12, 12),
        # a long prompt with a skewed expert load
        _ffn("q4_k_prefill_4096", 4096, 2048, 768, 128, 8, 12, 12, bf16=True, zipf=True),
        # Q4_K gate / up with Q5_1 down, the other mix that converted models hold, as an engine with its own router calls it
        _ffn("q4_k_q5_1_layer_4", 4, 2560, 640, 128, 8, 12, 7, kind="layer"),
        # the large layer with group-limited routing and a Q8_0 shared expert: a serving batch and a long prompt
        _ffn("large_decode_64", 64, 7168, 2048, 256, 8, 12, 12, bf16=True, groups=8, shared=True),
        _ffn("large_prefill_8192", 8192, 7168, 2048, 256, 8, 12, 12, bf16=True, groups=8, shared=True),
        # the dense block: single-stream decode, a batch of eight, a prompt
        _dense("dense_decode_1", 1, 5120, 17408),
        _dense("dense_decode_8", 8, 5120, 17408),
        _dense("dense_prefill_512", 512, 5120, 17408),
    ]


def _log(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    what = rng.choice(["q4", "q4", "q8", "mixed", "large", "dense"])
    bf16 = rng.random() < 0.5
    if what == "q4":
        c = _ffn("", _log(rng, 1, 4096), 256 * rng.randint(4, 16), 256 * rng.randint(2, 6), rng.choice([32, 60, 64, 96, 128, 160]), rng.choice([2, 4, 6, 8]), 12, 12,
                 bf16=bf16, zipf=rng.random() < 0.5)
    elif what == "q8":
        c = _ffn("", _log(rng, 1, 512), 256 * rng.randint(4, 16), 256 * rng.randint(2, 6), rng.choice([16, 32, 48, 64]), rng.choice([2, 4, 6]), 8, 8, bf16=bf16)
    elif what == "mixed":
        c = _ffn("", _log(rng, 1, 512), 256 * rng.randint(4, 16), 32 * rng.randint(16, 48), rng.choice([32, 60, 64, 128]), rng.choice([2, 4, 6, 8]), rng.choice([12, 13]),
                 rng.choice([7, 8]), kind="layer")
    elif what == "large":
        c = _ffn("", _log(rng, 1, 4096), 256 * rng.randint(16, 28), 256 * rng.randint(4, 8), rng.choice([64, 128, 256]), 8, 12, 12, bf16=True, groups=8, shared=True)
    else:
        c = _dense("", _log(rng, 1, 1024), 256 * rng.randint(8, 28), 256 * rng.randint(16, 72), rng.choice([12, 12, 8]), bf16=bf16)
    del c["name"]
    return c


def _tensor(gen, kind, rows, width):
    """rows x width weights as GGUF blocks: uniform quants and sub-scales, fp16 factors |N(0, 1)| of a trained tensor's size."""
    values, size = BLOCK[kind]
    n = rows * (width // values)
    if kind == 8:
        b = torch.randint(-127, 128, (n, size), generator=gen, device="cuda", dtype=torch.int8).view(torch.uint8)
        factors = [(0, 0.01, True)]
    else:
        b = torch.empty(n * size // 4, dtype=torch.int32, device="cuda").random_(-2**31, 2**31 - 1, generator=gen).view(torch.uint8).view(n, size)
        factors = {12: [(0, 0.01 / 32, True), (2, 0.01 / 32, True)], 13: [(0, 0.01 / 64, True), (2, 0.01 / 64, True)],
                   7: [(0, 0.01 / 16, True), (2, 0.01 / 2, False)]}[kind]
    for at, scale, positive in factors:
        d = torch.randn(n, generator=gen, device="cuda")
        d = (d.abs() if positive else d).mul_(scale).half()
        b[:, at:at + 2] = d.view(torch.uint8).view(n, 2)
    return b.view(-1)


def _experts(gen, c, experts):
    return (_tensor(gen, c["gate"], experts * c["inter"], c["hidden"]), _tensor(gen, c["gate"], experts * c["inter"], c["hidden"]),
            _tensor(gen, c["down"], experts * c["hidden"], c["inter"]))


def _zipf_bias(seed, experts):
    rank = np.random.default_rng(seed).permutation(experts) + 1.0
    p = rank ** -1.1
    return np.log(p / p.sum()).astype(np.float32)


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    H, E = c["hidden"], c.get("experts", 1)
    x = torch.randn((c["rows"], H), generator=gen, device="cuda")
    if c["bf16"]:
        x = x.bfloat16()
    gate, up, down = _experts(gen, c, E)
    s = {"case": c, "x": x}
    shape = ops.make_shape(H, c["inter"], E, c.get("top_k", 1), c["gate"], c["down"])
    if c["kind"] == "dense":
        s.update(shape=shape, gate=gate, up=up, down=down)
        return s
    router = torch.randn((E, H), generator=gen, device="cuda").mul_(0.02)
    bias = torch.from_numpy(_zipf_bias(seed, E)).cuda() if c["zipf"] else None
    policy = ops.sigmoid_group_policy(E, c["top_k"], c["groups"], c["groups"] // 2) if c["groups"] else ops.softmax_policy(E, c["top_k"])
    form = {"combine_form": b200moe.COMBINE_PARTS, "parts": 8 if c["groups"] else 2} if c["groups"] or c["gate"] == 8 else {"combine_form": b200moe.COMBINE_FMA_SLOTS}
    if c["kind"] == "layer":
        s.update(policy=policy, router=router, norm=torch.rand(H, generator=gen, device="cuda").add_(0.5),
                 layer=ops.MoeLayer(shape, gate, up, down, capacity=c["rows"], **form))
        return s
    select = torch.randn(E, generator=gen, device="cuda").mul_(0.1) if c["groups"] else None
    s["ffn"] = ops.MoeFfn(shape, policy, gate, up, down, router, capacity=c["rows"], logit_bias=bias, select_bias=select, **form)
    if c["shared"]:
        t = dict(c, gate=SHARED_TYPE, down=SHARED_TYPE)
        s["shared"] = (ops.make_shape(H, c["inter"], 1, 1, SHARED_TYPE, SHARED_TYPE),) + _experts(gen, t, 1)
    return s


def run(state):
    s = state
    x = s["x"]
    kind = s["case"]["kind"]
    if kind == "dense":
        return ops.enqueue_dense_ffn(s["shape"], s["gate"], s["up"], s["down"], ops.enqueue_quantize_a8(x))
    if kind == "layer":
        y, a8 = ops.enqueue_rmsnorm_a8(x, s["norm"])
        _, _, ids, weights = ops.enqueue_router(s["policy"], x=y, weight=s["router"])
        out, out_bf16 = s["layer"](a8, ids, weights, bf16=True)
        return {"ids": ids, "y": out, "y_bf16": out_bf16}
    shared = None
    if s["case"]["shared"]:
        shared = ops.enqueue_dense_ffn(*s["shared"], ops.enqueue_quantize_a8(x))
    return s["ffn"](x, shared=shared)


def _union(c):
    """How many distinct experts a window of such rows selects: the selection rule on random logits of the same spread."""
    if c["kind"] == "dense":
        return 1
    rng, E, k = np.random.default_rng(0), c["experts"], c["top_k"]
    logits = rng.standard_normal((c["rows"], E), dtype=np.float32) * np.float32(0.02 * math.sqrt(c["hidden"]))
    if c["zipf"]:
        logits += _zipf_bias(0, E)
    if c["groups"]:
        logits = 1.0 / (1.0 + np.exp(-logits)) + rng.standard_normal(E, dtype=np.float32) * np.float32(0.1)
        g = logits.reshape(c["rows"], c["groups"], -1)
        best = np.sort(g, axis=2)[:, :, -2:].sum(axis=2)
        dropped = np.argsort(best, axis=1)[:, : c["groups"] - c["groups"] // 2]
        np.put_along_axis(g, dropped[:, :, None], -np.inf, axis=1)
    return len(np.unique(np.argpartition(logits, E - k, axis=1)[:, E - k:]))


def _matrix_bytes(kind, rows, width):
    values, size = BLOCK[kind]
    return rows * (width // values) * size


def work(case):
    c = case
    R, H, inter = c["rows"], c["hidden"], c["inter"]
    n = _union(c)
    size = n * (2 * _matrix_bytes(c["gate"], inter, H) + _matrix_bytes(c["down"], H, inter)) + R * H * ((2 if c["bf16"] else 4) + 4)
    flops = 6.0 * R * c.get("top_k", 1) * H * inter
    if c["kind"] != "dense":
        size += c["experts"] * H * 4
        flops += 2.0 * R * c["experts"] * H
        if c["shared"]:
            size += 2 * _matrix_bytes(SHARED_TYPE, inter, H) + _matrix_bytes(SHARED_TYPE, H, inter)
            flops += 6.0 * R * H * inter
        if c["kind"] == "layer":
            size += R * H * 2
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """Every operation of the path has a declared order and rounding (integer dots, single-precision chains), so two correct
    implementations give the same bits."""
    return "exact"
