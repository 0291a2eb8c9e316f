"""The workloads this framework is timed on, each one pass through the public entry points
(``mc.compile`` once, then ``prog(...)`` per call).

Four families, all over the sizes the repository's builders, tests and benchmark use:

* ``mlp``      the MLP block (RMS norm, gate/up + SwiGLU, down + residual), forward, 1 .. 4096 rows
* ``decode``   one token per sequence of a 1B-shaped Llama: 1 .. 64 sequences, contexts 256 .. 16384,
               one shared position or one per sequence (ragged), the token ids gathered inside the launch
               (``fused``) or embedded by the caller
* ``prefill``  prompts of 64 .. 4096 tokens through decoder layers and the lm_head of the last token
* ``dit``      adaLN-Zero blocks over 1 .. 32 images of 64 or 256 tokens

Weights are bf16 with the scale of a trained model's initialisation, embeddings come from the tied
lm_head, caches hold N(0, 1) rows up to each sequence's position.  Every pass starts from the same
state: the caller sets the position (and token) of the step it asks for, as a batching server does,
so that a pass can be repeated.
"""

from __future__ import annotations

import math

import torch

import megacute_b200 as mc
from megacute_b200 import workloads as W
from megacute_b200.builders import dit_stack, llama_decode, llama_stack, mlp_block

LLAMA = W.LLAMA_1B
# (heads, kv heads) per head dimension: the same width, cache row and parameter count either way
HEADS = {64: (32, 8), 128: (16, 4)}
DIT = dict(E=1024, H=16, F=4096)
MLP = dict(E=2048, F=5632)

# Largest amounts of work of a family, which draw() keeps to.
MAX_MLP_ROWS = 4096
MAX_CACHE_ROWS = 64 * 4096
MAX_PROMPT_TOKENS = 4 * 4096
MAX_IMAGES = 32


def listed() -> list[dict]:
    return [
        # one token through one block: the smallest call, latency of the launch and of two dependent linears
        {"name": "mlp_1", "kind": "mlp", "rows": 1},
        # a decode batch's worth of tokens through one block: the benchmark's MLP configuration
        {"name": "mlp_256", "kind": "mlp", "rows": 256},
        # an odd number of prompt tokens through one block: large GEMMs with a ragged last tile
        {"name": "mlp_3001", "kind": "mlp", "rows": 3001},
        # interactive chat, one user: the benchmark's headline step
        {"name": "decode_b1_1k", "kind": "decode", "batch": 1, "ctx": 1024, "head_dim": 64, "ragged": False, "fused": True},
        # one user with a long document in context
        {"name": "decode_b1_16k", "kind": "decode", "batch": 1, "ctx": 16384, "head_dim": 64, "ragged": False, "fused": True},
        # a lightly loaded server: a few sequences of different lengths, sampling left to the caller
        {"name": "decode_b5_ragged", "kind": "decode", "batch": 5, "ctx": 2900, "head_dim": 64, "ragged": True, "fused": False},
        # a loaded server with short contexts
        {"name": "decode_b64_1k", "kind": "decode", "batch": 64, "ctx": 1024, "head_dim": 64, "ragged": False, "fused": True},
        # a loaded server with longer contexts: the KV cache dominates
        {"name": "decode_b64_4k", "kind": "decode", "batch": 64, "ctx": 4096, "head_dim": 64, "ragged": False, "fused": False},
        # time to first token of one short prompt of odd length, whole model
        {"name": "prefill_1x333", "kind": "prefill", "batch": 1, "seq": 333, "head_dim": 64, "layers": 16},
        # a batch of long prompts (the benchmark's prefill shape; a quarter of its identical layers)
        {"name": "prefill_4x4096", "kind": "prefill", "batch": 4, "seq": 4096, "head_dim": 64, "layers": 4},
        # prompts through layers with 128-wide heads
        {"name": "prefill_2x2048_d128", "kind": "prefill", "batch": 2, "seq": 2048, "head_dim": 128, "layers": 4},
        # one denoising step for a batch of images: the benchmark's DiT configuration
        {"name": "dit_32", "kind": "dit", "images": 32, "tokens": 256, "blocks": 28},
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """An integer of [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["mlp", "decode", "decode", "prefill", "prefill", "dit"])
    if kind == "mlp":
        return {"kind": kind, "rows": _spread(rng, 2, MAX_MLP_ROWS)}
    if kind == "decode":
        batch = _spread(rng, 1, 64)
        ctx = _spread(rng, 256, min(16384, MAX_CACHE_ROWS // batch))
        return {"kind": kind, "batch": batch, "ctx": ctx, "head_dim": rng.choice([64, 64, 64, 128]),
                "ragged": rng.random() < 0.4, "fused": rng.random() < 0.5}
    if kind == "prefill":
        seq = _spread(rng, 64, 4096)
        batch = _spread(rng, 1, max(1, min(16, MAX_PROMPT_TOKENS // seq)))
        return {"kind": kind, "batch": batch, "seq": seq, "head_dim": rng.choice([64, 64, 64, 128]), "layers": 4}
    return {"kind": kind, "images": _spread(rng, 1, MAX_IMAGES), "tokens": rng.choice([64, 256]), "blocks": 28}


def _llama(case) -> dict:
    """E, H, KVH, F, n, vocab of the case's model (n: decode steps run the whole model)."""
    h, kvh = HEADS[case["head_dim"]]
    return dict(E=LLAMA["E"], H=h, KVH=kvh, F=LLAMA["F"], n=case.get("layers", LLAMA["n"]), vocab=LLAMA["vocab"])


def _max_seq(ctx: int) -> int:
    """Cache rows per sequence: room for at least 64 more tokens, in whole attention tiles."""
    return (ctx + 64 + 127) // 128 * 128


def _positions(case) -> list[int]:
    """Tokens already in the cache of each sequence: all the same, or spread evenly from a sixteenth
    of the context to all of it."""
    b, ctx = case["batch"], case["ctx"]
    if not case["ragged"]:
        return [ctx] * b
    lo = max(1, ctx // 16)
    return [ctx if b == 1 else lo + (ctx - lo) * i // (b - 1) for i in range(b)]


def _bound(prog, tensors: dict) -> dict:
    """The tensors a program binds (weights made for a whole model can be more)."""
    names = {b.name for b in prog.g.inputs + prog.g.params + prog.g.states}
    return {k: v for k, v in tensors.items() if k in names}


def prepare(case: dict, seed: int) -> dict:
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "mlp":
        g = mlp_block(case["rows"], MLP["E"], MLP["F"])
        tensors = W.mlp_block_inputs(case["rows"], MLP["E"], MLP["F"], seed, dev)
    elif kind == "dit":
        g = dit_stack(case["images"], case["tokens"], DIT["E"], DIT["H"], DIT["F"], case["blocks"])
        tensors = W.dit_inputs(case["images"], case["tokens"], DIT["E"], DIT["F"], case["blocks"], seed, dev)
    else:
        m = _llama(case)
        dims = (m["E"], m["H"], m["KVH"], m["F"], m["n"])
        weights = W.llama_weights(*dims, m["vocab"], seed, dev)
        gen = torch.Generator(device=dev).manual_seed(seed + 1)
        if kind == "prefill":
            b, s = case["batch"], case["seq"]
            g = llama_stack(b, s, *dims, eps=LLAMA["eps"], vocab=m["vocab"])
            cos, sin = W.rope_tables(s, case["head_dim"], LLAMA["theta"], dev)
            ids = torch.randint(0, m["vocab"], (b * s,), generator=gen, device=dev)
            tensors = dict(x=weights["lm_head"][ids], cos=cos, sin=sin, **weights)
        else:
            b, max_seq = case["batch"], _max_seq(case["ctx"])
            g = llama_decode(b, *dims, max_seq, m["vocab"], LLAMA["eps"], fused_step=case["fused"], ragged=case["ragged"])
            st, ids = W.llama_decode_state(b, *dims[:3], m["n"], max_seq, case["ctx"], m["vocab"], seed + 1, dev)
            cos, sin = W.rope_tables(max_seq, case["head_dim"], LLAMA["theta"], dev)
            pos = _positions(case)
            start = torch.tensor(pos if case["ragged"] else pos[:1], dtype=torch.int32, device=dev).reshape(-1, 1)
            if case["ragged"]:
                start = start[torch.randperm(b, generator=gen, device=dev)].contiguous()
            tensors = dict(cos=cos, sin=sin, ids=ids.to(torch.int32).reshape(b, 1), **weights, **st)
            tensors["pos"] = start.clone()
            prog = mc.compile(g)
            return {"kind": kind, "fused": case["fused"], "prog": prog, "args": _bound(prog, tensors), "start": start,
                    "tokens": ids.to(torch.int32).reshape(b, 1) if case["fused"] else ids, "table": weights["lm_head"]}
    prog = mc.compile(g)
    return {"kind": kind, "prog": prog, "args": _bound(prog, tensors)}


def run(state: dict):
    args = state["args"]
    if state["kind"] != "decode":
        return state["prog"](**args)
    # the step's token and position go in, as they do for every step of a batching server
    args["pos"].copy_(state["start"])
    if state["fused"]:
        args["ids"].copy_(state["tokens"])
    else:
        torch.index_select(state["table"], 0, state["tokens"], out=args["x"])
    logits = state["prog"](**args)
    # (a fused step also leaves the greedy ids: the argmax of these logits, not compared on their own because two logits
    # of random weights can be equal in bf16)
    return {"logits": logits, "pos": args["pos"], "k_cache": args["k_cache"], "v_cache": args["v_cache"]}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "mlp":
        m, e, f = case["rows"], MLP["E"], MLP["F"]
        return {"bytes": 2 * (3 * e * f + e + 2 * m * e), "flops": 6 * m * e * f}
    if kind == "dit":
        b, s, n, e, f = case["images"], case["tokens"], case["blocks"], DIT["E"], DIT["F"]
        layer_params = 6 * e * e + 6 * e + 4 * e * e + 4 * e + 2 * e * f + f + e
        flops = n * (2 * b * 6 * e * e + 2 * b * s * (4 * e * e + 2 * e * f) + 4 * b * s * s * e)
        return {"bytes": 2 * (n * layer_params + 2 * b * s * e + b * e), "flops": flops}
    m = _llama(case)
    e, f, d, n, vocab = m["E"], m["F"], case["head_dim"], m["n"], m["vocab"]
    kv = m["KVH"] * d
    layer_mats = e * (e + 2 * kv) + e * e + 3 * e * f
    params = n * (layer_mats + 2 * e) + e + vocab * e
    b = case["batch"]
    if kind == "prefill":
        s = case["seq"]
        pairs = s * (s + 1) // 2
        flops = n * (2 * b * s * layer_mats + 4 * b * pairs * m["H"] * d) + 2 * b * e * vocab
        return {"bytes": 2 * (params + b * s * e + 2 * s * d + b * vocab), "flops": flops}
    tokens = sum(_positions(case))
    flops = n * (2 * b * layer_mats + 4 * (tokens + b) * m["H"] * d) + 2 * b * e * vocab
    # weights once, the cached rows of every layer once, the new rows, logits
    return {"bytes": 2 * (params + n * 2 * kv * (tokens + b) + b * e + b * vocab), "flops": flops}


def tolerance(case: dict) -> dict:
    # bf16 weights, bf16 results and 16-bit private activations over up to 28 layers; positions are whole numbers
    return {"rel": 1e-2}
