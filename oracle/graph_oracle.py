"""TEST INFRASTRUCTURE -- the CPU/fp32 oracle for megakernel graphs.  Not part of the product.

Only ``tests/``, ``__graft_entry__.smoke()`` and the ``cpu_baseline`` / ``--impl reference`` legs of
``bench.py`` may import this file; the runtime package never does.

What it is: an fp32 torch interpreter of an *un-rewritten* op graph (no pass, no tiling, no
fusion).  It restates the op semantics the reference documents on its op dataclasses and kernels:

    Linear / swiglu      megacute/graph.py:118-122, megacute/ops/gemm.py:280-316
    SplitFinalize        megacute/graph.py:177
    Unary / activations  megacute/dmath.py:37-56   (gelu and gelu_tanh are both the tanh form)
    Binary               megacute/graph.py:214-226, megacute/dmath.py:59-70
    SwiGLU               megacute/graph.py:239
    Modulate             megacute/graph.py:259
    Norm                 megacute/graph.py:281, megacute/ops/norm.py:94-114
    Rope                 megacute/graph.py:306-307, megacute/ops/eltwise.py:146-180
    Attention            megacute/graph.py:333-335, megacute/ops/attention.py:303-305
    RopeAppend           megacute/graph.py:375-379
    DecodeAttention      megacute/graph.py:412-418
    Increment            megacute/graph.py:472
    Gather / Argmax      (no graph op in the reference) the torch calls around its launch, examples/llama/llama1b.py:103-105

Pinning: the reference ships no tests, golden vectors or fixtures for this path, and its device
code cannot run in the build container (it needs nvidia-cutlass-dsl 4.8.0 and a Blackwell GPU), so
the float parity is UNPINNED by reference outputs.  What is pinned instead (tests/test_oracle.py):
every op of this file against an independent torch formulation (torch.nn.functional); the
graph structure / swiglu_weight permutation against fixtures generated by importing the
reference's host code (tests/golden/); and the reading of the ops only the reference's passes make
(LinearSplit, SplitFinalize, Linear with a folded rms_eps over a derived weight, RopeAppend over a
split-K workspace, the fused DecodeAttention) by evaluating graphs rewritten by the REFERENCE's own
fold_norms / split_k / fuse_rope_attention / split_kv (megacute/runtime.py:44-199) and requiring
the result of the un-rewritten graph (tests/golden/ref_passes.pt).

The interpreter is duck-typed: it accepts graphs built by this repository's ``Graph`` or by the
reference's (ops expose ``kind`` and the same operand names).  Intermediate buffers are fp32;
``state`` tensors keep their own dtype so a value appended to a bf16 cache is read back rounded,
as on the device.
"""

from __future__ import annotations

import math

import torch

F32 = torch.float32


def act_fn(name, x):
    if name is None or name == "identity":
        return x
    if name == "relu":
        return torch.relu(x)
    if name == "silu":
        return x * torch.sigmoid(x)
    if name == "sigmoid":
        return torch.sigmoid(x)
    if name in ("gelu", "gelu_tanh"):
        return 0.5 * x * (1.0 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x * x * x)))
    if name == "exp":
        return torch.exp(x)
    if name == "neg":
        return -x
    if name == "square":
        return x * x
    raise ValueError(f"unknown activation {name}")


def binary_fn(name, a, b):
    return {"add": torch.add, "sub": torch.sub, "mul": torch.mul, "max": torch.maximum, "min": torch.minimum}[name](a, b)


def rotate_half(x, cos, sin, D):
    """x: (..., heads*D) rows; cos/sin: (..., D) broadcastable per row."""
    lead = x.shape[:-1]
    xh = x.reshape(*lead, -1, D)
    x1, x2 = xh[..., :D // 2], xh[..., D // 2:]
    c, s = cos.unsqueeze(-2), sin.unsqueeze(-2)
    o1 = x1 * c[..., :D // 2] - x2 * s[..., :D // 2]
    o2 = x2 * c[..., D // 2:] + x1 * s[..., D // 2:]
    return torch.cat([o1, o2], -1).reshape(*lead, -1)


class Evaluator:
    def __init__(self, g, tensors: dict, device="cpu"):
        self.g = g
        self.dev = torch.device(device)
        self.vals: dict[int, torch.Tensor] = {}
        named = {b.name: b for b in list(g.inputs) + list(g.params) + list(g.states)}
        for name, b in named.items():
            t = tensors[name].to(self.dev)
            assert tuple(t.shape) == (b.rows, b.cols), (name, t.shape)
            if b.kind == "state":
                self.vals[b.id] = t.clone()
            else:
                self.vals[b.id] = t            # read only: upcast lazily per view
        self.state_names = {b.name: b for b in g.states}

    # ---- view access
    def derived(self, b):
        """A norm-folded weight made by the reference's fold_norms: rows [r0, r0 + n) of the source
        times the norm gain in fp32, rounded to the buffer's dtype (megacute/runtime.py:344-354)."""
        d = torch.zeros(b.rows, b.cols, dtype=b.dtype, device=self.dev)
        for src, r0, n, gv in b.derive:
            gain = self.vals[gv.buf.id][gv.row0:gv.row0 + 1, gv.col0:gv.col0 + gv.cols].to(F32)
            d[r0:r0 + n] = (self.vals[src.id][r0:r0 + n].to(F32) * gain).to(b.dtype)
        return d

    def rd(self, v):
        if v is None:
            return None
        if v.buf.id not in self.vals and v.buf.kind == "derived":
            self.vals[v.buf.id] = self.derived(v.buf)
        if v.buf.id not in self.vals and v.buf.kind == "workspace":      # zero on entry to a launch
            b = v.buf
            self.vals[b.id] = torch.zeros(b.rows, b.cols, dtype=torch.int32 if b.dtype == torch.int32 else F32,
                                          device=self.dev)
        t = self.vals[v.buf.id]
        return t[v.row0:v.row0 + v.rows, v.col0:v.col0 + v.cols].to(F32)

    def wr(self, v, val):
        b = v.buf
        if b.id not in self.vals:
            dt = b.dtype if b.kind == "state" else (torch.int32 if b.dtype == torch.int32 else F32)
            self.vals[b.id] = torch.zeros(b.rows, b.cols, dtype=dt, device=self.dev)
        t = self.vals[b.id]
        t[v.row0:v.row0 + v.rows, v.col0:v.col0 + v.cols] = val.to(t.dtype)

    def pos_of(self, v):
        return int(self.vals[v.buf.id][v.row0, v.col0])

    def pos_rows(self, v, batch):
        """Position of every sequence: one shared value, or (repo extension) one row of pos per sequence."""
        col = self.vals[v.buf.id][v.row0:v.row0 + v.rows, v.col0]
        return [int(col[b if v.rows > 1 else 0]) for b in range(batch)]

    # ---- ops
    def run(self):
        for op in self.g.ops:
            getattr(self, "op_" + op.kind)(op)
        outs = [self.rd(v) for v in self.g.outputs]
        states = {name: self.vals[b.id] for name, b in self.state_names.items()}
        return outs, states

    def op_Linear(self, o):
        x = self.rd(o.x)
        if getattr(o, "rms_eps", None) is not None:     # a norm folded by a pass (not in user graphs)
            x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + o.rms_eps)
            nw = self.rd(getattr(o, "norm_w", None))
            if nw is not None:
                x = x * nw
        y = x @ self.rd(o.w).T
        if o.act == "swiglu":
            N = y.shape[1]
            y = y.reshape(-1, N // 128, 2, 64)
            y = (act_fn("silu", y[:, :, 0]) * y[:, :, 1]).reshape(-1, N // 2)
        else:
            if o.bias is not None:
                y = y + self.rd(o.bias)
            y = act_fn(o.act, y)
            if getattr(o, "gate", None) is not None:    # (this repository's fused form: a gated residual)
                y = y * self.rd(o.gate).repeat_interleave(o.gate_group, 0)
            if o.residual is not None:
                y = y + self.rd(o.residual)
            if getattr(o, "cos", None) is not None:     # (this repository's fused form: the first rope_cols columns rotated)
                p = torch.arange(y.shape[0], device=self.dev) % o.seq
                n = o.rope_cols
                y = torch.cat([rotate_half(y[:, :n], self.rd(o.cos)[p], self.rd(o.sin)[p], o.head_dim), y[:, n:]], 1)
        self.wr(o.out, y)

    def op_LinearSplit(self, o):
        x = self.rd(o.x)
        if getattr(o, "rms_eps", None) is not None:     # megacute/graph.py:154-158: rms_eps as in Linear
            x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + o.rms_eps)
        self.wr(o.ws, self.rd(o.ws) + x @ self.rd(o.w).T)

    def op_SplitFinalize(self, o):
        y = self.rd(o.ws)
        if o.bias is not None:
            y = y + self.rd(o.bias)
        y = act_fn(o.act, y)
        if getattr(o, "gate", None) is not None:        # (this repository's fused form: a gated residual)
            y = y * self.rd(o.gate).repeat_interleave(o.gate_group, 0)
        if o.residual is not None:
            y = y + self.rd(o.residual)
        self.wr(o.out, y)
        self.wr(o.ws, torch.zeros_like(y))

    def op_Unary(self, o):
        self.wr(o.out, act_fn(o.fn, self.rd(o.x)))

    def op_Binary(self, o):
        b = self.rd(o.b).repeat_interleave(o.b_group, 0)
        if getattr(o, "gate", None) is not None:        # (this repository's fused form: b is gated per row group first)
            b = b * self.rd(o.gate).repeat_interleave(o.gate_group, 0)
        self.wr(o.out, binary_fn(o.fn, self.rd(o.a), b))

    def op_SwiGLU(self, o):
        self.wr(o.out, act_fn(o.act, self.rd(o.gate)) * self.rd(o.up))

    def op_Modulate(self, o):
        sc = self.rd(o.scale).repeat_interleave(o.group, 0)
        sh = self.rd(o.shift).repeat_interleave(o.group, 0)
        self.wr(o.out, self.rd(o.x) * (1.0 + sc) + sh)

    def op_Norm(self, o):
        x = self.rd(o.x)
        if o.rms:
            y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + o.eps)
        else:
            mu = x.mean(-1, keepdim=True)
            var = (x * x).mean(-1, keepdim=True) - mu * mu
            y = (x - mu) * torch.rsqrt(var + o.eps)
        if o.weight is not None:
            y = y * self.rd(o.weight)
        if o.bias is not None:
            y = y + self.rd(o.bias)
        if getattr(o, "scale", None) is not None:       # (this repository's fused form: adaLN modulation of the normalised rows)
            y = y * (1.0 + self.rd(o.scale).repeat_interleave(o.group, 0)) + self.rd(o.shift).repeat_interleave(o.group, 0)
        self.wr(o.out, y)

    def op_Rope(self, o):
        x = self.rd(o.x)
        p = torch.arange(x.shape[0], device=self.dev) % o.seq
        self.wr(o.out, rotate_half(x, self.rd(o.cos)[p], self.rd(o.sin)[p], o.head_dim))

    def op_Attention(self, o):
        B, H, KVH, D = o.batch, o.heads, o.kv_heads, o.head_dim
        q = self.rd(o.q).reshape(B, o.seq_q, H, D).transpose(1, 2)
        k = self.rd(o.k).reshape(B, o.seq_k, KVH, D).transpose(1, 2).repeat_interleave(H // KVH, 1)
        v = self.rd(o.v).reshape(B, o.seq_k, KVH, D).transpose(1, 2).repeat_interleave(H // KVH, 1)
        out = torch.empty(B, H, o.seq_q, D, dtype=F32, device=self.dev)
        for b in range(B):                     # per batch entry to bound the score matrix
            s = (q[b] @ k[b].transpose(-1, -2)) * o.scale
            if o.causal:
                mask = torch.ones(o.seq_q, o.seq_k, dtype=torch.bool, device=self.dev).tril()
                s = s.masked_fill(~mask, float("-inf"))
            out[b] = torch.softmax(s, -1) @ v[b]
        self.wr(o.out, out.transpose(1, 2).reshape(B * o.seq_q, H * D))

    def op_RopeAppend(self, o):
        H, KVH, D, L = o.heads, o.kv_heads, o.head_dim, o.max_seq
        qkv = self.rd(o.qkv)
        B = qkv.shape[0]
        ps = self.pos_rows(o.pos, B)
        idx = torch.tensor(ps, device=self.dev)
        cos, sin = self.rd(o.cos)[idx], self.rd(o.sin)[idx]          # one table row per sequence
        self.wr(o.q_out, rotate_half(qkv[:, :H * D], cos, sin, D))
        kr = rotate_half(qkv[:, H * D:(H + KVH) * D], cos, sin, D)
        for b in range(B):
            self.wr(o.k_cache.rows_slice(b * L + ps[b], 1), kr[b:b + 1])
            self.wr(o.v_cache.rows_slice(b * L + ps[b], 1), qkv[b:b + 1, (H + KVH) * D:])
        if o.qkv.buf.kind == "workspace":               # an fp32 split-K workspace is read, then zeroed (graph.py:379-380)
            self.wr(o.qkv, torch.zeros_like(qkv))

    def op_DecodeAttention(self, o):
        B, H, KVH, D, L = o.batch, o.heads, o.kv_heads, o.head_dim, o.max_seq
        G = H // KVH
        ps = self.pos_rows(o.pos, B)
        window = int(getattr(o, "window", 0) or 0)
        q = self.rd(o.q)
        if getattr(o, "k_new", None) is not None:       # a RopeAppend fused in by a pass (not in user graphs)
            idx = torch.tensor(ps, device=self.dev)
            cos, sin = self.rd(o.cos)[idx], self.rd(o.sin)[idx]
            q = rotate_half(q, cos, sin, D)
            kr = rotate_half(self.rd(o.k_new), cos, sin, D)
            vn = self.rd(o.v_new)
            for b in range(B):
                self.wr(o.k_cache.rows_slice(b * L + ps[b], 1), kr[b:b + 1])
                self.wr(o.v_cache.rows_slice(b * L + ps[b], 1), vn[b:b + 1])
            if o.q.buf.kind == "workspace":             # "An fp32 QKV row is a split-K workspace: the op zeroes what it read"
                for v_ in (o.q, o.k_new, o.v_new):
                    self.wr(v_, torch.zeros(v_.rows, v_.cols, device=self.dev))
        q = q.reshape(B, KVH, G, D)
        kc = self.vals[o.k_cache.buf.id]
        vc = self.vals[o.v_cache.buf.id]
        r0, c0 = o.k_cache.row0, o.k_cache.col0
        kall = kc[r0:r0 + B * L, c0:c0 + KVH * D].reshape(B, L, KVH, D)
        r0, c0 = o.v_cache.row0, o.v_cache.col0
        vall = vc[r0:r0 + B * L, c0:c0 + KVH * D].reshape(B, L, KVH, D)
        out = torch.empty(B, KVH, G, D, dtype=F32, device=self.dev)
        if len(set(ps)) == 1 and not window:            # the reference's case: one position for the batch, the whole context
            p = ps[0]
            k, v = kall[:, :p + 1], vall[:, :p + 1]
            step = max(1, (1 << 26) // max(1, (p + 1) * KVH * D))
            for b0 in range(0, B, step):
                kk = k[b0:b0 + step].to(F32).permute(0, 2, 1, 3)        # (b, KVH, keys, D)
                vv = v[b0:b0 + step].to(F32).permute(0, 2, 1, 3)
                s = (q[b0:b0 + step] @ kk.transpose(-1, -2)) * o.scale
                out[b0:b0 + step] = torch.softmax(s, -1) @ vv
        else:                                           # per sequence: rows [max(0, pos + 1 - window), pos]
            for b in range(B):
                lo = max(0, ps[b] + 1 - window) if window else 0
                kk = kall[b, lo:ps[b] + 1].to(F32).permute(1, 0, 2)     # (KVH, keys, D)
                vv = vall[b, lo:ps[b] + 1].to(F32).permute(1, 0, 2)
                s = (q[b] @ kk.transpose(-1, -2)) * o.scale
                out[b] = torch.softmax(s, -1) @ vv
        self.wr(o.out, out.reshape(B, H * D))

    def op_Gather(self, o):
        """out[r] = table[ids[r, 0]] (the torch index_select of the reference's step, examples/llama/llama1b.py:103-104)."""
        ids = self.vals[o.ids.buf.id][o.ids.row0:o.ids.row0 + o.ids.rows, o.ids.col0].long()
        tab = self.vals[o.table.buf.id][o.table.row0:o.table.row0 + o.table.rows, o.table.col0:o.table.col0 + o.table.cols]
        self.wr(o.out, tab[ids].to(F32))              # (rows first: the table is the whole embedding matrix)

    def op_Argmax(self, o):
        """ids[r, 0] = argmax(x[r]), first maximum (torch's argmax, examples/llama/llama1b.py:105)."""
        t = self.vals[o.ids.buf.id]
        t[o.ids.row0:o.ids.row0 + o.ids.rows, o.ids.col0] = self.rd(o.x).argmax(-1).to(t.dtype)

    def op_Increment(self, o):
        t = self.vals[o.pos.buf.id]
        t[o.pos.row0:o.pos.row0 + o.pos.rows, o.pos.col0] += 1


def evaluate(g, tensors: dict, device="cpu"):
    """Run graph ``g`` on named tensors.  Returns (outputs: list of fp32 tensors in ``g.outputs``
    order, states: dict name -> updated state tensor in its own dtype)."""
    return Evaluator(g, tensors, device).run()


def rel_l2(a: torch.Tensor, ref: torch.Tensor) -> float:
    a, ref = a.to(torch.float64), ref.to(torch.float64)
    return float((a - ref).norm() / ref.norm().clamp_min(1e-30))


def rope_tables(max_seq: int, D: int, theta: float = 500000.0, dtype=torch.bfloat16):
    """Rotate-half cos/sin tables (max_seq, D), fp64 math, no frequency scaling
    (examples/llama/llama1b.py:59-71 without the llama3 scaling branch)."""
    inv = 1.0 / theta ** (torch.arange(0, D, 2, dtype=torch.float64) / D)
    ang = torch.arange(max_seq, dtype=torch.float64)[:, None] * inv[None]
    ang = torch.cat([ang, ang], -1)
    return ang.cos().to(dtype).contiguous(), ang.sin().to(dtype).contiguous()
