"""Edges of the tile shapes: 256-row GEMM tiles and their epilogues, uneven K splits, rotated heads in a linear's
epilogue, the two-tile prefill attention, norms of many rows per instruction -- against the fp32 oracle."""
import pytest
import torch

import megacute_b200 as mc
from megacute_b200 import passes
from megacute_b200 import workloads as W
from oracle.graph_oracle import evaluate, rel_l2
from tests.helpers import TOL
from tests.test_gpu_ops import rnd, run_both

F32, BF = torch.float32, torch.bfloat16
# one rounding of an fp32 value to bf16: at most 2^-9 of it, so at most 2^-9 in rel-L2; 5 % for fp32 sums of K <= 2048
# products (K 2^-24) and the approximate exponentials of the activations (2^-20)
ONE_ROUNDING = 1.05 * 2.0 ** -9


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,plan,kw", [
    (129, 256, 64, (1, 256, 256), {}),                                          # one k-tile, one row in the lower half
    (256, 128, 192, (1, 256, 128), {"bias": True}),
    (257, 384, 256, (1, 256, 128), {"res": BF}),                                # a second row tile of one row
    (300, 512, 2048, (1, 256, 256), {"act": "gelu_tanh", "bias": True}),
    (300, 256, 320, (1, 256, 128), {"act": "relu"}),
    (400, 512, 128, (1, 256, 256), {"act": "swiglu"}),
    (385, 256, 448, (1, 256, 256), {"res": F32}),
    (513, 256, 64, (1, 256, 256), {"res": BF, "act": "silu"}),                  # (activation in front of a residual)
    (320, 512, 256, (1, 256, 256), {"gate": 64}),                               # gated residual, 64 rows per gate row
    (320, 128, 256, (1, 256, 128), {"gate": 40}),                               # (a warp's rows span two gate rows)
    (320, 256, 256, (1, 128, 128), {"gate": 64}),                               # ... in 128-row tiles
    (192, 136, 192, (1, 128, 128), {"gate": 3, "bias": True}),                  # (a gate row per three rows, a last step of eight columns)
    (400, 264, 64, (1, 128, 128), {"gate": 40, "gres": F32}),
    (96, 1000, 128, (1, 128, 128), {"gate": 32, "act": "silu"}),
    (600, 256, 320, (3, 256, 128), {"bias": True}),                             # 5 k-tiles in 3 splits
    (200, 256, 448, (4, 128, 128), {"act": "relu"}),                            # 7 in 4, 128 x 128 tiles
    (320, 1000, 448, (4, 128, 128), {"gate": 64}),                              # ... finished with a gated residual
    (300, 136, 448, (3, 128, 128), {"gate": 3, "bias": True, "act": "silu", "gres": F32, "gdt": F32}),
    (200, 520, 448, (2, 128, 128), {"bias": True, "act": "gelu_tanh", "res": BF}),
    (135, 264, 448, (3, 128, 128), {"bias": True, "res": F32}),                 # (ragged in both directions, finished with a residual)
    (150, 136, 96, (1, 128, 128), {}),                                          # K of whole 32s: the mma.sync body
])
def test_tile_epilogues(cuda, monkeypatch, M, N, K, plan, kw):
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: plan if a[4] > 1 else (1, *plan[1:]))
    g = mc.Graph()
    n_out = N // 2 if kw.get("act") == "swiglu" else N
    x, w = g.input("x", (M, K)), g.param("w", (N, K))
    t = {"x": rnd((M, K), 1.0, 1), "w": rnd((N, K), K ** -0.5, 2)}
    bias = res = None
    if kw.get("bias"):
        bias, t["b"] = g.param("b", (1, n_out)), rnd((1, n_out), 0.5, 3)
    if kw.get("res"):
        res, t["r"] = g.input("r", (M, n_out), kw["res"]), rnd((M, n_out), 1.0, 4).to(kw["res"])
    y = g.linear(x, w, bias=bias, act=kw.get("act"), residual=res)
    if kw.get("gate"):
        r, gate = g.input("r", (M, N), kw.get("gres", BF)), g.input("gate", (M // kw["gate"], N), kw.get("gdt", BF))
        t["r"], t["gate"] = rnd((M, N), 1.0, 4).to(kw.get("gres", BF)), rnd((M // kw["gate"], N), 1.0, 5).to(kw.get("gdt", BF))
        y = g.add(r, g.binary(y, gate, "mul", b_group=kw["gate"]))
    g.output(y)
    outs, ref, _, _, prog = run_both(g, t, cuda, steps=2)                       # twice: split-K workspaces are zeroed again
    for a, b in zip(outs, ref):
        assert rel_l2(a, b) < ONE_ROUNDING
    if kw.get("gate"):
        assert not any(o.kind == "Binary" for o in prog.g.ops)
    if plan[0] == 1:
        lin = [o for o in prog.g.ops if o.kind == "Linear"][0]
        assert (lin.bm or 128, lin.bn or 128) == plan[1:] and prog.tcgen05_ops == (1 if K % 64 == 0 else 0)
        assert (lin.gate is not None) == bool(kw.get("gate"))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [9, 15, 16, 17, 31, 33, 56, 57, 64, 65, 120, 121, 127])
def test_activation_copies_of_the_rows_there_are(cuda, M):
    """128 x 128 tiles copy a ragged op's activation rows in whole groups of eight; what the rest of a stage holds -- another op's
    rows, not numbers here -- reaches no output."""
    g = mc.Graph()
    y = g.linear(g.input("z", (128, 1024)), g.param("v", (20480, 1024)))         # every SM's stages filled with values that are not numbers
    h = g.linear(g.input("x", (M, 1024)), g.param("w", (19000, 1024)), act="gelu_tanh")
    g.output(y)
    g.output(h)
    t = {"z": torch.full((128, 1024), float("nan"), dtype=torch.bfloat16), "v": rnd((20480, 1024), 0.03, 3),
         "x": rnd((M, 1024), 1.0, 1), "w": rnd((19000, 1024), 0.03, 2)}
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert prog.tcgen05_ops == 2 and outs[0].isnan().all()
    assert torch.isfinite(outs[1]).all() and rel_l2(outs[1], ref[1]) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(9, 128, 64), (32, 136, 64), (33, 128, 128), (63, 264, 192), (97, 128, 64), (128, 8, 128)])
@pytest.mark.parametrize("res,act", [(BF, None), (F32, None), (BF, "silu"), (None, "gelu_tanh"), (None, None), (F32, "gelu_tanh"), (F32, "silu"), (None, "silu"),
                                     (BF, "relu"), (None, "relu")])
def test_row_groups_of_an_epilogue(cuda, M, N, K, res, act):
    """Rows that end anywhere in a warp's groups of four, one accumulator (one k-tile) or two, columns that end inside a tile."""
    g = mc.Graph()
    t = {"x": rnd((M, K), 1.0, 1), "w": rnd((N, K), K ** -0.5, 2), "b": rnd((1, N), 0.5, 3), "r": rnd((M, N), 1.0, 4).to(res or BF)}
    y = g.linear(g.input("x", (M, K)), g.param("w", (N, K)), bias=g.param("b", (1, N)), act=act, residual=g.input("r", (M, N), res) if res else None)
    g.output(y)
    outs, ref, _, _, prog = run_both(g, t if res else {k: v for k, v in t.items() if k != "r"}, cuda)
    assert prog.tcgen05_ops == 1 and rel_l2(outs[0], ref[0]) < ONE_ROUNDING


@pytest.mark.gpu
@pytest.mark.parametrize("M", [9, 31, 32, 33, 100])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "relu"])
def test_activation_and_a_private_residual(cuda, M, act):
    """An activation in front of a 16-bit private residual, on both sides of the number of rows that go through shared memory."""
    g = mc.Graph()
    y = g.linear(g.input("x", (M, 128)), g.param("v", (192, 128)))
    y = g.linear(y, g.param("w", (192, 192)), act=act, residual=y) if M == 100 else g.linear(y, g.param("w", (192, 192)), act=act, residual=y, bias=g.param("b", (1, 192)))
    g.output(g.linear(y, g.param("u", (64, 192))))
    t = {"x": rnd((M, 128), 1.0, 1), "v": rnd((192, 128), 0.1, 2), "w": rnd((192, 192), 0.1, 3), "u": rnd((64, 192), 0.1, 4), "b": rnd((1, 192), 0.5, 5)}
    outs, ref, *_ = run_both(g, t if M != 100 else {k: v for k, v in t.items() if k != "b"}, cuda)
    assert rel_l2(outs[0], ref[0]) < 1.6 * 2.0 ** -9          # (rounding of the output to bf16 2^-9, of two activations to fp16 2^-12 each, tanh.approx 2^-11)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,H,KVH,D,K", [(1, 130, 1, 1, 64, 64), (5, 30, 3, 1, 64, 128), (3, 3, 2, 2, 64, 64), (1, 128, 1, 1, 128, 64), (2, 65, 4, 2, 128, 192)])
def test_rotated_heads_at_tile_edges(cuda, B, S, H, KVH, D, K):
    """128 x 128 tiles whose last one is half empty or holds rotated and other heads, sequences that wrap inside a warp's rows."""
    g = mc.Graph()
    x, w = g.input("x", (B * S, K)), g.param("w", ((H + 2 * KVH) * D, K))
    cos, sin = g.input("cos", (S, D)), g.input("sin", (S, D))
    qkv = g.linear(x, w)
    q = g.rope(qkv.cols_slice(0, H * D), cos, sin, heads=H, head_dim=D, seq=S)
    k = g.rope(qkv.cols_slice(H * D, KVH * D), cos, sin, heads=KVH, head_dim=D, seq=S)
    g.output(g.attention(q, k, qkv.cols_slice((H + KVH) * D, KVH * D), batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=True))
    cs, sn = W.rope_tables(S, D)
    t = {"x": rnd((B * S, K), 1.0, 1), "w": rnd(((H + 2 * KVH) * D, K), 0.1, 2), "cos": cs, "sin": sn}
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert not any(o.kind == "Rope" for o in prog.g.ops) and prog.tcgen05_ops == 1
    assert rel_l2(outs[0], ref[0]) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,kw", [(1024, 4096, 64, {"res": F32}), (1024, 4160, 64, {"act": "gelu_tanh"}), (2000, 3080, 128, {"res": BF, "act": "silu"}),
                                      (64, 40960, 64, {"res": BF})])
def test_direct_epilogues_one_behind_the_other(cuda, monkeypatch, M, N, K, kw):
    """Several 128 x 128 tiles per CTA whose epilogues have no barrier of their own, of one and two k-tiles: the state of the next one changes
    while warps without a part in the products may still be at this one's start.  Many launches, the same bits."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 128, 128))
    g = mc.Graph()
    t = {"x": rnd((M, K), 1.0, 1), "w": rnd((N, K), K ** -0.5, 2)}
    if kw.get("res"):
        t["r"] = rnd((M, N), 1.0, 3).to(kw["res"])
    g.output(g.linear(g.input("x", (M, K)), g.param("w", (N, K)), act=kw.get("act"), residual=g.input("r", (M, N), kw["res"]) if kw.get("res") else None))
    dev = {n: u.to(cuda) for n, u in t.items()}
    prog = mc.compile(g)
    assert -(-M // 128) * -(-N // 128) > 148 and [o.kind for o in prog.g.ops] == ["Linear"]
    got = prog(**dev).clone()
    assert prog.tcgen05_ops == 1 and rel_l2(got, evaluate(g, dev, cuda)[0][0]) < ONE_ROUNDING
    for _ in range(200):
        y = prog(**dev)
    assert torch.equal(y, got)
    prog.check()


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [8, 40, 72])
@pytest.mark.parametrize("B,S,H,KVH,D,K", [(1, 100, 2, 1, 64, 64), (3, 50, 1, 1, 64, 128), (1, 100, 2, 1, 128, 64), (2, 129, 1, 1, 128, 192), (1, 9, 3, 1, 64, 64)])
def test_columns_behind_rotated_heads(cuda, B, S, H, KVH, D, K, extra):
    """A projection with more behind v than whole heads: rows end inside a warp's piece of columns.  Nothing reaches the next row's first
    head or, behind the last row, the memory after the buffer."""
    n, heads = (H + 2 * KVH) * D, H + KVH
    g = mc.Graph()
    x, w = g.input("x", (B * S, K)), g.param("w", (n + extra, K))
    cos, sin = g.input("cos", (S, D)), g.input("sin", (S, D))
    y = g.linear(x, w)
    q = g.rope(y.cols_slice(0, H * D), cos, sin, heads=H, head_dim=D, seq=S)
    k = g.rope(y.cols_slice(H * D, KVH * D), cos, sin, heads=KVH, head_dim=D, seq=S)
    g.output(g.attention(q, k, y.cols_slice(heads * D, KVH * D), batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=True))
    g.output(g.unary(y.cols_slice(n, extra), "silu"))
    cs, sn = W.rope_tables(S, D)
    t = {"x": rnd((B * S, K), 1.0, 1), "w": rnd((n + extra, K), 0.1, 2), "cos": cs, "sin": sn}
    prog = mc.compile(g)
    lin = [o for o in prog.g.ops if o.kind == "Linear"][0]
    assert lin.cos is not None and not any(o.kind == "Rope" for o in prog.g.ops)
    buf = lin.out.buf
    guarded = torch.full((buf.rows * buf.cols + 1024,), 7.0, dtype=buf.dtype, device=cuda)
    prog._bufs[buf.id] = guarded[:buf.rows * buf.cols].view(buf.rows, buf.cols)
    ref, _ = evaluate(g, t)
    for _ in range(3):
        outs = prog(**{name: v.to(cuda) for name, v in t.items()})
        prog.check()
        assert prog.tcgen05_ops == 1 and (guarded[buf.rows * buf.cols:] == 7.0).all()
        for o, r in zip(outs, ref):
            assert rel_l2(o, r.to(cuda)) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("B,S,D,tile", [(1, 150, 64, (128, 128)), (3, 50, 128, (128, 128)), (2, 129, 64, (256, 256)), (1, 257, 128, (256, 128)),
                                        (1, 300, 128, (256, 256))])
def test_rotated_heads(cuda, monkeypatch, B, S, D, tile, tcgen05):
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, *tile))
    if not tcgen05:
        monkeypatch.setenv("MEGACUTE_B200_NO_TCGEN05", "1")
    H, KVH, K = 2, 1, 192
    g = mc.Graph()
    x, w = g.input("x", (B * S, K)), g.param("w", ((H + 2 * KVH) * D, K))
    cos, sin = g.input("cos", (S, D)), g.input("sin", (S, D))
    qkv = g.linear(x, w)
    q = g.rope(qkv.cols_slice(0, H * D), cos, sin, heads=H, head_dim=D, seq=S)
    k = g.rope(qkv.cols_slice(H * D, KVH * D), cos, sin, heads=KVH, head_dim=D, seq=S)
    g.output(g.attention(q, k, qkv.cols_slice((H + KVH) * D, KVH * D), batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=True))
    cs, sn = W.rope_tables(S, D)
    t = {"x": rnd((B * S, K), 1.0, 1), "w": rnd(((H + 2 * KVH) * D, K), 0.1, 2), "cos": cs, "sin": sn}
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert not any(o.kind == "Rope" for o in prog.g.ops)
    assert rel_l2(outs[0], ref[0]) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("B,Sq,Sk,H,KVH,D,causal", [
    (1, 1, 1, 1, 1, 64, False), (2, 128, 128, 2, 1, 64, True), (1, 129, 129, 3, 1, 64, True), (1, 255, 640, 2, 2, 64, False),
    (3, 257, 257, 2, 1, 64, True), (1, 385, 385, 4, 2, 64, True), (1, 700, 65, 2, 1, 64, False),
    (1, 64, 300, 1, 1, 128, False), (2, 130, 130, 2, 1, 128, True), (1, 520, 520, 3, 1, 128, True), (1, 256, 1000, 2, 2, 128, False),
])
def test_prefill_attention_tiles(cuda, B, Sq, Sk, H, KVH, D, causal):
    """Odd numbers of query tiles and key blocks, one tile only, masked and ragged last blocks.  (A CTA has one instruction at most
    here; several of them: test_attention_instructions_follow_one_another_on_a_cta.)"""
    g = mc.Graph()
    q, k, v = g.input("q", (B * Sq, H * D)), g.input("k", (B * Sk, KVH * D)), g.input("v", (B * Sk, KVH * D))
    a = g.attention(q, k, v, batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=causal)
    b = g.attention(a, k, v, batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=causal)
    g.output(a, b)
    t = {"q": rnd((B * Sq, H * D), 2.0, 1), "k": rnd((B * Sk, KVH * D), 2.0, 2), "v": rnd((B * Sk, KVH * D), 1.0, 3)}
    outs, ref, _, _, prog = run_both(g, t, cuda, steps=2)
    assert prog.tcgen05_attention_ops == 2
    for x, y in zip(outs, ref):
        assert rel_l2(x, y) < TOL


def rows_close(outs, ref):
    """Every row on its own: a damaged tile or head does not hide in the norm of the whole tensor."""
    for o, want in zip(outs, ref):
        err = (o.float() - want).norm(dim=1) / want.norm(dim=1)
        assert torch.isfinite(err).all() and float(err.max()) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [(64, 64), (128, 128), (64, 128), (128, 64)])
def test_attention_instructions_follow_one_another_on_a_cta(cuda, monkeypatch, first, second):
    """Two to four attention instructions per SM and op, so that barriers, K and V stages, score buffers and O change hands between
    instructions, from one head size to the other, and with what else uses the ring and the work area: 256-row tiles, streaming
    linears, 128-row tiles, norms of several rows per warp."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256) if a[1] % 256 == 0 else (1, 128, 128))
    monkeypatch.setattr(passes, "hoist_linears", lambda g: g)
    B, S = 16, 350                                            # two instructions per (sequence, head), the second with 94 queries
    g = mc.Graph()
    x, x1 = g.input("x", (B * S, 256)), g.input("x1", (1, 256))
    t = {"x": rnd((B * S, 256), 1.0, 1), "x1": rnd((1, 256), 1.0, 2)}

    def w(rows, cols):
        name = f"w{len(t)}"
        # (q, k and v of standard deviation 1/2, scores of 1/4 and at most about 2: the roundings of q and k, 2^-9 each, move a softmax
        # weight by less than 2^-7.  So no row collects more than a few 16-bit roundings per block, 3e-3 to 5e-3 over the three)
        t[name] = rnd((rows, cols), 0.5 * cols ** -0.5, len(t))
        return g.param(name, (rows, cols))

    y = x
    for n, D in enumerate((first, second, first)):
        H, KVH = 1024 // D, 512 // D
        qkv = g.linear(y, w(2048, 256))
        q, k, v = qkv.cols_slice(0, 1024), qkv.cols_slice(1024, 512), qkv.cols_slice(1536, 512)
        a = g.attention(q, k, v, batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=n != 1)
        b = g.attention(a, k, v, batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=n == 1)
        g.output(a, b, g.linear(x1, w(148 * 16, 256)))
        y = g.rms_norm(g.linear(g.linear(b, w(1024 + 128, 1024)), w(256, 1024 + 128)))
    g.output(y)
    prog = mc.compile(g)
    att = [e - s for o, (s, e) in zip(prog.g.ops, prog.sched.node_ranges) if o.kind == "Attention"]
    assert len(att) == 6 and min(att) > 1.7 * prog.sm_count             # (head_dim 128: 256 instructions, 64: 512)
    dev = {n: u.to(cuda) for n, u in t.items()}
    ref, _ = evaluate(g, dev, cuda)
    for _ in range(3):
        rows_close(prog(**dev), ref)
    prog.check()
    assert prog.tcgen05_attention_ops == 6


@pytest.mark.gpu
def test_tile_kinds_follow_one_another_on_a_cta(cuda, monkeypatch):
    """256 x 256, 256 x 128 and 128 x 128 tiles in turns, two and more of each per SM, with one k-tile and with more k-tiles than there
    are stages: each kind divides the same memory in its own way, and loads and MMAs of the next tile run ahead."""
    plans = {2560: (1, 256, 256), 2432: (1, 256, 128), 1280: (1, 128, 128)}
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: plans[a[1]])
    monkeypatch.setattr(passes, "hoist_linears", lambda g: g)
    M = 4001                                                  # (the last row tile: 161 rows)
    g = mc.Graph()
    x, t = g.input("x", (M, 576)), {"x": rnd((M, 576), 1.0, 1)}
    xs = {64: x.cols_slice(0, 64), 576: x}
    order = [(2560, 64), (2432, 64), (2560, 576), (2432, 576), (1280, 576), (2432, 64), (2432, 576), (1280, 64), (2560, 576), (2560, 64)]
    for i, (N, K) in enumerate(order):
        t[f"w{i}"], t[f"b{i}"] = rnd((N, K), K ** -0.5, 10 + i), rnd((1, N), 0.5, 30 + i)
        g.output(g.linear(xs[K], g.param(f"w{i}", (N, K)), bias=g.param(f"b{i}", (1, N)), act="relu" if i % 3 else None))
    prog = mc.compile(g)
    assert all((o.bm or 128, o.bn or 128) == plans[N][1:] for o, (N, _) in zip(prog.g.ops, order))
    assert [e - s for s, e in prog.sched.node_ranges][:2] == [160, 304]
    dev = {n: u.to(cuda) for n, u in t.items()}
    ref, _ = evaluate(g, dev, cuda)
    for _ in range(5):
        rows_close(prog(**dev), ref)
    prog.check()
    assert prog.tcgen05_ops == len(order)


HALVED = [  # rows, columns, K, residual type, gate group -> row blocks of the two linears (three quarters of 148 SMs: 111 tiles)
    (2500, 2048, 4160, F32, 0, (2, 8)), (2700, 2560, 4160, BF, 0, (8, 3)), (920, 7168, 4160, None, 0, None), (700, 9216, 4160, None, 0, (2, 1)),
    (640, 9216, 4160, None, 0, None), (2560, 2048, 4160, BF, 64, (2, 8)), (2600, 2048, 4160, F32, 40, None), (2500, 2048, 4096, F32, 0, None),
    (3600, 2048, 4160, F32, 0, None),
]


def halved_graph(M, N, K, rdt, group, front=None):
    """The linear behind another one of K outputs and `front` (as many as it has itself) columns."""
    front = front or N
    g, t = mc.Graph(), {"x": rnd((M, front), 1.0, 1), "v": rnd((K, front), front ** -0.5, 5), "w": rnd((N, K), K ** -0.5, 2)}
    y = g.linear(g.linear(g.input("x", (M, front)), g.param("v", (K, front))), g.param("w", (N, K)))
    if rdt:
        t["r"] = rnd((M, N), 1.0, 3).to(rdt)
        if group:
            t["gate"] = rnd((M // group, N), 1.0, 4)
            y = g.binary(y, g.input("gate", (M // group, N)), "mul", b_group=group)
        y = g.add(g.input("r", (M, N), rdt), y)
    g.output(y)
    return g, t


@pytest.mark.parametrize("M,N,K,rdt,group,blocks", HALVED)
def test_which_linears_end_in_half_tiles(monkeypatch, M, N, K, rdt, group, blocks):
    """The two linears cover the rows once, with the operands' rows beside them."""
    monkeypatch.delenv("MEGACUTE_B200_WIDE_TILES", raising=False)
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256) if a[1] == N else (1, 128, 128))
    halves = lambda **kw: [o for o in passes.run_all(halved_graph(M, N, K, rdt, group, **kw)[0], 148).ops if o.kind == "Linear" and o.w.buf.name == "w"]
    assert len(halves(front=N - 8)) == 1                       # (not behind a shorter one; alone: below)
    ops = halves()
    if blocks is None:
        assert len(ops) == 1 and ops[0].bn == 256
        return
    a, b = ops
    assert (a.bn, b.bn, -(-a.x.rows // 256), -(-b.x.rows // 256)) == (256, 128, *blocks) and a.x.rows + b.x.rows == M
    assert a.x.rows == 256 * blocks[0] and a.w.same(b.w)
    for f in ("x", "out", "residual"):
        u, v = getattr(a, f), getattr(b, f)
        assert (u is None) == (v is None) and (u is None or (u.row0, v.row0, u.rows, v.rows) == (0, a.x.rows, a.x.rows, b.x.rows))
    if group:
        assert (a.gate.rows, b.gate.row0, b.gate.rows) == (a.x.rows // group, a.x.rows // group, b.x.rows // group)


def test_a_linear_of_the_launchs_inputs_keeps_whole_tiles(monkeypatch):
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256))
    g = mc.Graph()
    g.output(g.linear(g.input("x", (2500, 4160)), g.param("w", (2048, 4160))))
    assert [o.bn for o in passes.run_all(g, 148).ops] == [256]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,rdt,group,blocks", [c for c in HALVED if c[-1]])
def test_half_tiles_of_the_last_rows(cuda, monkeypatch, M, N, K, rdt, group, blocks):
    """The same bits as whole tiles give (every output is summed over K in the same order), and the oracle's values."""
    monkeypatch.delenv("MEGACUTE_B200_WIDE_TILES", raising=False)
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256) if a[1] == N else (1, 128, 128))
    g, t = halved_graph(M, N, K, rdt, group)
    dev = {n: u.to(cuda) for n, u in t.items()}
    prog = mc.compile(g)
    assert [o.bn for o in prog.g.ops if o.kind == "Linear" and o.w.buf.name == "w"] == [256, 128]
    got = prog(**dev).clone()
    prog.check()
    monkeypatch.setattr(passes, "halve_last_tiles", lambda g, sm_count: g)
    whole = mc.compile(g)
    assert [o.bn for o in whole.g.ops if o.kind == "Linear" and o.w.buf.name == "w"] == [256]
    assert torch.equal(got, whole(**dev))
    ref, _ = evaluate(g, dev, cuda)
    assert rel_l2(got, ref[0]) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("tcgen05", [True, False])
@pytest.mark.parametrize("S,D,causal", [(64, 64, False), (64, 128, True), (100, 64, True), (129, 64, False), (200, 128, False), (300, 64, True), (257, 128, True), (7, 64, True)])
def test_attention_of_sequences_beside_one_that_is_not_numbers(cuda, monkeypatch, S, D, causal, tcgen05):
    """Keys and values behind a sequence's last one are the next sequence's (or not written yet): they have no weight, whatever they are."""
    if not tcgen05:
        monkeypatch.setenv("MEGACUTE_B200_ATTN_TCGEN05", "0")
    B, H, KVH = 4, 4, 2
    g = mc.Graph()
    q, k, v = g.input("q", (B * S, H * D)), g.input("k", (B * S, KVH * D)), g.input("v", (B * S, KVH * D))
    g.output(g.attention(q, k, v, batch=B, heads=H, kv_heads=KVH, head_dim=D, causal=causal))
    t = {"q": rnd((B * S, H * D), 1.0, 1), "k": rnd((B * S, KVH * D), 1.0, 2), "v": rnd((B * S, KVH * D), 1.0, 3)}
    ref, _ = evaluate(g, t)
    t["k"][S:2 * S], t["v"][S:2 * S], t["v"][3 * S:] = float("nan"), float("nan"), float("inf")
    prog = mc.compile(g)
    out = prog(**{n: u.to(cuda) for n, u in t.items()}).float().cpu()
    prog.check()
    assert prog.tcgen05_attention_ops == (1 if tcgen05 else 0)
    for b in (0, 2):
        assert rel_l2(out[b * S:(b + 1) * S], ref[0][b * S:(b + 1) * S]) < TOL
    assert not torch.isfinite(out[S:2 * S]).any() and not torch.isfinite(out[3 * S:]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [-0.3, 0.0])
@pytest.mark.parametrize("D", [64, 128])
def test_prefill_attention_scale_not_positive(cuda, D, scale):
    """A negative scale turns the order of the scores around; zero gives every unmasked key the same weight."""
    S, H = 200, 2
    g = mc.Graph()
    q, k, v = (g.unary(g.input(n, (S, H * D)), "identity") for n in "qkv")       # (private tensors: fp16)
    g.output(g.attention(q, k, v, batch=1, heads=H, head_dim=D, causal=True, scale=scale))
    t = {n: rnd((S, H * D), 1.0, i) for i, n in enumerate("qkv")}
    outs, ref, _, _, prog = run_both(g, t, cuda, steps=2)
    assert rel_l2(outs[0], ref[0]) < TOL and prog.tcgen05_attention_ops == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,dtype,rms,group", [
    (257, 2048, BF, True, 0), (1190, 1024, BF, True, 0), (2390, 1000, BF, False, 0), (3001, 2048, F32, True, 0), (2400, 1024, BF, False, 40),
    (9600, 256, BF, True, 0), (2500, 8, F32, True, 0), (1201, 2040, BF, False, 0), (1999, 1504, F32, False, 0),
])
def test_norm_many_rows(cuda, rows, cols, dtype, rms, group):
    """8, 16, 24 and 64 rows per instruction, a last instruction with fewer, modulation rows that change inside one."""
    g = mc.Graph()
    x = g.input("x", (rows, cols), dtype)
    t = {"x": rnd((rows, cols), 2.0, 1, 0.3).to(dtype)}
    y = g.rms_norm(x, g.param("w", (1, cols))) if rms else g.layer_norm(x)
    if rms:
        t["w"] = rnd((1, cols), 0.1, 2, 1.0)
    if group:
        n = rows // group
        y = g.modulate(y, g.input("sc", (n, cols)), g.input("sh", (n, cols)), group=group)
        t["sc"], t["sh"] = rnd((n, cols), 0.3, 3), rnd((n, cols), 0.3, 4)
    g.output(y)
    outs, ref, *_ = run_both(g, t, cuda)
    assert rel_l2(outs[0], ref[0]) < ONE_ROUNDING


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,dtype,group,mod", [
    (300, 72, F32, 3, F32), (1200, 1000, BF, 8, BF), (1208, 1024, F32, 604, F32), (2400, 264, BF, 1, BF), (261, 2048, F32, 0, BF), (2403, 1032, BF, 0, BF),
    (9602, 520, F32, 0, BF), (149, 2048, F32, 0, BF), (150, 1000, BF, 0, BF), (64, 1024, F32, 32, BF), (12, 264, BF, 3, BF), (3, 1024, BF, 1, F32),
    (5001, 2048, BF, 0, BF), (5500, 1032, F32, 0, BF), (1500, 1024, F32, 3, F32), (9602, 520, BF, 2, BF), (2403, 1024, BF, 1, F32), (301, 8, F32, 1, BF), (1200, 72, BF, 4, BF),
    (64, 1152, F32, 64, BF), (150, 1032, BF, 2, F32), (256, 1024, F32, 256, BF), (200, 4096, BF, 0, BF), (256, 2056, F32, 0, BF),
])
def test_norm_shares_gain_and_modulation(cuda, rows, cols, dtype, group, mod):
    """Gain and modulation in shared memory: several groups per instruction, a group per row, both types, warps without a row."""
    g = mc.Graph()
    x = g.input("x", (rows, cols), dtype)
    t = {"x": rnd((rows, cols), 2.0, 1, 0.3).to(dtype)}
    if group:
        n = rows // group
        y = g.modulate(g.layer_norm(x), g.input("sc", (n, cols), mod), g.input("sh", (n, cols), mod), group=group)
        t["sc"], t["sh"] = rnd((n, cols), 0.3, 3).to(mod), rnd((n, cols), 0.3, 4).to(mod)
    else:
        y, t["w"] = g.rms_norm(x, g.param("w", (1, cols))), rnd((1, cols), 0.1, 2, 1.0)
    g.output(y)
    outs, ref, *_ = run_both(g, t, cuda)
    assert rel_l2(outs[0], ref[0]) < ONE_ROUNDING


def test_hoisted_linears_keep_their_order():
    """A linear moves behind the op it depends on and in front of unrelated ones only; what reads or overwrites its operands stays put."""
    g = mc.Graph()
    c, w = g.input("c", (32, 64)), g.param("w", (64, 64))
    s = g.unary(c, "silu")
    x = g.input("x", (32, 64))
    for _ in range(6):
        x = g.add(x, g.unary(x, "relu"))
    late = g.linear(s, w)
    near = g.linear(x, w)
    g.output(g.add(g.add(x, late), near))
    ops = passes.hoist_linears(g).ops
    assert [o.kind for o in ops[:2]] == ["Unary", "Linear"] and ops[1].x.same(s)
    seen = {b.id for b in g.inputs + g.params}
    for o in ops:
        assert all(v.buf.id in seen for v in o.reads)
        seen |= {v.buf.id for v in o.writes}
    assert len(ops) == len(g.ops) and ops[-3].x.same(x)


@pytest.mark.gpu
def test_ring_changes_hands_behind_256_row_tiles(cuda, monkeypatch):
    """The epilogues of 256-row tiles leave a bias row, gate rows or staged rows in the ring's memory; 128-row tiles and streaming
    linears that depend on nothing follow at once, with copies into the same bytes.  Every SM has each of them, three times over."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 128))
    monkeypatch.setattr(passes, "hoist_linears", lambda g: g)                   # (keeps the order below)
    M, N, K, Ns = 2048, 2432, 64, 148 * 128
    g = mc.Graph()
    x, xs, x1 = g.input("x", (M, K)), g.input("xs", (100, K)), g.input("x1", (1, K))
    t = {"x": rnd((M, K), 1.0, 1), "xs": rnd((100, K), 1.0, 2), "x1": rnd((1, K), 1.0, 3)}

    def p(name, rows, cols, std):
        t[name] = rnd((rows, cols), std, len(t))
        return g.param(name, (rows, cols))

    for i in range(3):
        a = g.linear(x, p(f"wa{i}", N, K, 0.1), bias=p(f"ba{i}", 1, N, 1.0), act="relu")
        s = g.linear(xs, p(f"ws{i}", Ns, K, 0.1))
        r = g.temp((M, N))
        g.unary(a, "identity", out=r)
        b = g.add(r, g.binary(g.linear(x, p(f"wb{i}", N, K, 0.1)), p(f"gb{i}", M // 64, N, 1.0), "mul", b_group=64))
        v = g.linear(x1, p(f"wv{i}", Ns, K, 0.1))
        c = g.linear(x, p(f"wc{i}", N, K, 0.1), act="relu", residual=a)
        s2 = g.linear(xs, p(f"wt{i}", Ns, K, 0.1))
        g.output(a, s, b, v, c, s2)
    prog = mc.compile(g)
    dev = {k: w.to(cuda) for k, w in t.items()}
    ref, _ = evaluate(g, dev, cuda)
    for _ in range(10):
        rows_close(prog(**dev), ref)
    prog.check()
    assert sum(o.kind == "Linear" and o.bm == 256 for o in prog.g.ops) == 9
