"""GPU parity tests: every op kind of the megakernel against the fp32 oracle, through the C ABI.

Floating point: bf16 outputs within rel-L2 <= 1e-2 of the fp32 evaluation (helpers.TOL).
Integer work (pos, cache rows written, counters): bit exact.
"""
import numpy as np
import pytest
import torch

import megacute_b200 as mc
from megacute_b200 import config as C, passes
from megacute_b200 import workloads as W
from oracle.graph_oracle import evaluate, rel_l2
from tests.helpers import TOL, small_decode, to_cpu

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def rnd(shape, std=1.0, seed=0, mean=0.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * std + mean).to(BF)


def run_both(g, tensors, cuda, steps=1, **kw):
    """Run graph g on the GPU (steps launches) and in the oracle; return (gpu outs, oracle outs, gpu
    states, oracle states, prog)."""
    prog = mc.compile(g, **kw)
    dev = {k: v.to(cuda).contiguous() for k, v in tensors.items()}
    ref_t = {k: v.clone() for k, v in tensors.items()}
    outs = ref = None
    states = {b.name for b in g.states}
    for _ in range(steps):
        outs = prog(**dev)
        outs = outs if isinstance(outs, tuple) else (outs,)
        ref, st = evaluate(g, ref_t)
        for n in states:
            ref_t[n] = st[n]
    prog.check()
    return [o.float().cpu() for o in outs], ref, {n: dev[n].cpu() for n in states}, {n: ref_t[n] for n in states}, prog


def assert_close(outs, ref, tol=TOL):
    for o, r in zip(outs, ref):
        assert torch.isfinite(o).all()
        assert rel_l2(o, r) < tol, rel_l2(o, r)


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("rows,cols,rms,affine", [(1, 2048, True, True), (3, 512, True, False), (300, 1024, False, False),
                                                 (260, 256, False, True), (64, 2048, True, True)])
def test_norm(cuda, rows, cols, rms, affine):
    g = mc.Graph()
    x = g.input("x", (rows, cols))
    w = g.param("w", (1, cols)) if affine else None
    if rms:
        y = g.rms_norm(x, w, eps=1e-5)
    else:
        y = g.layer_norm(x, w, g.param("b", (1, cols)) if affine else None, eps=1e-5)
    g.output(g.unary(y, "identity"))         # keeps the norm unfolded and adds a dependent op
    t = {"x": rnd((rows, cols), 2.0, 1, 0.3)}
    if affine:
        t["w"] = rnd((1, cols), 0.1, 2, 1.0)
        if not rms:
            t["b"] = rnd((1, cols), 0.1, 3)
    outs, ref, *_ = run_both(g, t, cuda)
    assert_close(outs, ref)


@pytest.mark.parametrize("fn", ["relu", "silu", "gelu_tanh", "gelu", "exp", "neg", "sigmoid", "square", "identity"])
def test_unary(cuda, fn):
    g = mc.Graph()
    x = g.input("x", (70, 1032))
    g.output(g.unary(x, fn))
    outs, ref, *_ = run_both(g, {"x": rnd((70, 1032), 1.0, 4)}, cuda)
    assert_close(outs, ref)


@pytest.mark.parametrize("fn", ["add", "sub", "mul", "max", "min"])
def test_binary_and_broadcast(cuda, fn):
    g = mc.Graph()
    a = g.input("a", (96, 520))
    b = g.input("b", (96, 520))
    c = g.input("c", (3, 520))
    y = g.binary(a, b, fn)
    g.output(y, g.binary(y, c, fn, b_group=32))
    outs, ref, *_ = run_both(g, {"a": rnd((96, 520), 1, 5), "b": rnd((96, 520), 1, 6), "c": rnd((3, 520), 1, 7)}, cuda)
    assert_close(outs, ref)


def test_swiglu_modulate_rope(cuda):
    g = mc.Graph()
    S, H, D = 40, 6, 64
    x = g.input("x", (2 * S, H * D))
    u = g.input("u", (2 * S, H * D))
    sc = g.input("sc", (2, H * D))
    sh = g.input("sh", (2, H * D))
    cos = g.input("cos", (S, D))
    sin = g.input("sin", (S, D))
    a = g.swiglu(x, u)
    b = g.modulate(x, sc, sh, group=S)
    c = g.rope(x, cos, sin, heads=H, head_dim=D, seq=S)
    d = g.rope(x.cols_slice(128, 256), cos, sin, heads=4, head_dim=D, seq=S)      # a column slice of a wider buffer
    g.output(a, b, c, d)
    cs, sn = W.rope_tables(S, D)
    t = {"x": rnd((2 * S, H * D), 1, 8), "u": rnd((2 * S, H * D), 1, 9), "sc": rnd((2, H * D), 0.3, 10),
         "sh": rnd((2, H * D), 0.3, 11), "cos": cs, "sin": sn}
    outs, ref, *_ = run_both(g, t, cuda)
    assert_close(outs, ref)


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("M,K,N,act,bias,res,norm", [
    (1, 2048, 512, None, False, False, False),
    (1, 2048, 3072, None, False, False, True),
    (1, 8192, 296, None, False, True, False),
    (1, 2048, 1024, "swiglu", False, False, True),
    (2, 4096, 640, "gelu_tanh", True, True, False),
    (4, 1024, 1000, "silu", True, False, True),
    (8, 2048, 1544, "relu", True, True, True),
    (3, 1064, 136, None, True, True, False),
    (5, 264, 256, "swiglu", False, False, False),
])
def test_streaming_linear(cuda, M, K, N, act, bias, res, norm):
    """Linears with <= 8 rows run on the weight-streaming path (GEMV)."""
    g = mc.Graph()
    x = g.input("x", (M, K))
    w = g.param("w", (N, K))
    n_out = N // 2 if act == "swiglu" else N
    h = g.rms_norm(x, g.param("nw", (1, K)), eps=1e-5) if norm else x
    y = g.linear(h, w, bias=g.param("b", (1, n_out)) if bias else None, act=act,
                 residual=g.input("r", (M, n_out)) if res else None)
    g.output(y)
    t = {"x": rnd((M, K), 1.0, 1), "w": rnd((N, K), 0.03, 2)}
    if norm:
        t["nw"] = rnd((1, K), 0.05, 3, 1.0)
    if bias:
        t["b"] = rnd((1, n_out), 0.5, 4)
    if res:
        t["r"] = rnd((M, n_out), 1.0, 5)
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert_close(outs, ref)
    assert [o.kind for o in prog.g.ops] == ["Linear"]                 # the norm was folded


def test_streaming_linear_chain_and_counters(cuda):
    """Dependent streaming linears; dependency counters end at arrivals * launches."""
    g = mc.Graph()
    x = g.input("x", (1, 512))
    w1 = g.param("w1", (1024, 512))
    w2 = g.param("w2", (512, 1024))
    w3 = g.param("w3", (2048, 512))
    h = g.linear(x, w1, act="silu")
    y = g.linear(h, w2, residual=x)
    g.output(g.linear(y, w3))
    t = {"x": rnd((1, 512), 1, 1), "w1": rnd((1024, 512), 0.04, 2), "w2": rnd((512, 1024), 0.03, 3),
         "w3": rnd((2048, 512), 0.04, 4)}
    outs, ref, _, _, prog = run_both(g, t, cuda, steps=3)
    assert_close(outs, ref)
    assert np.array_equal(prog.counters(), prog.sched.counter_target * 3)


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("B,H,KVH,D,max_seq,ctx", [(1, 8, 2, 64, 256, 100), (3, 4, 4, 64, 128, 0), (2, 8, 1, 128, 256, 200),
                                                  (1, 32, 8, 64, 1152, 1024), (20, 8, 2, 64, 384, 300),
                                                  (40, 16, 8, 64, 256, 129), (160, 4, 1, 64, 128, 0), (50, 8, 4, 128, 256, 77),
                                                  (150, 32, 8, 64, 128, 64)])
@pytest.mark.parametrize("fused", [False, True])
def test_decode_attention(cuda, B, H, KVH, D, max_seq, ctx, fused):
    """rope_append + decode_attention, kept separate (q_out is also an output) or fused by the pass."""
    _decode_attention_case(cuda, B, H, KVH, D, max_seq, ctx, fused)


@pytest.mark.parametrize("B,H,KVH,max_seq,ctx,splits", [
    (9, 8, 2, 128, 37, 1), (9, 8, 2, 128, 37, 2), (12, 16, 2, 256, 45, 3), (16, 32, 8, 384, 300, 1), (16, 32, 8, 384, 300, 5),
    (3, 32, 8, 256, 17, 4), (70, 32, 8, 128, 0, 2), (24, 8, 8, 256, 200, 3), (150, 32, 8, 256, 129, 2)])
@pytest.mark.parametrize("fused", [False, True])
def test_decode_attention_many_sequences(cuda, monkeypatch, B, H, KVH, max_seq, ctx, splits, fused):
    """The many-sequence form: one instruction = a sequence's KV split over all kv heads, whole cache rows
    through bulk copies, one warp per kv head.  GQA groups of 1, 4 and 8, fewer kv heads than warps,
    contexts that are not a multiple of the 16-row tile, shorter than one tile, or empty; splits that get
    no keys; the last split of a sequence to arrive merges."""
    monkeypatch.setenv("MEGACUTE_B200_ATT_BULK", "1")
    monkeypatch.setenv("MEGACUTE_B200_KV_SPLITS", str(splits))
    prog = _decode_attention_case(cuda, B, H, KVH, 64, max_seq, ctx, fused)
    att = [o for o in prog.g.ops if o.kind == "DecodeAttention"]
    assert att and all(o.bulk and o.heads_per_inst == KVH and o.splits == min(splits, max_seq // 64) for o in att)


@pytest.mark.parametrize("B,H,KVH,max_seq,ctx", [(40, 16, 8, 512, 300), (33, 8, 2, 256, 37), (64, 32, 8, 128, 0), (61, 32, 8, 384, 257), (150, 8, 8, 256, 129),
                                                 (16, 32, 8, 1024, 960)])
@pytest.mark.parametrize("fused", [False, True])
def test_decode_attention_equal_shares(cuda, monkeypatch, B, H, KVH, max_seq, ctx, fused):
    """The many-sequence form with ranges of keys of unequal length, one or two instructions per SM: contexts that leave many of them empty, that
    end inside a tile, splits of one sequence on several SMs and of several on one."""
    monkeypatch.setenv("MEGACUTE_B200_ATT_BULK", "1")
    monkeypatch.setattr(passes, "shares_pay", lambda *a: True)
    prog = _decode_attention_case(cuda, B, H, KVH, 64, max_seq, ctx, fused)
    att = [o for o in prog.g.ops if o.kind == "DecodeAttention"]
    assert att and all(o.shares and o.splits == max(x[4] for x in o.shares) for o in att)


def _decode_attention_case(cuda, B, H, KVH, D, max_seq, ctx, fused):
    g = mc.Graph()
    qkv = g.input("qkv", (B, (H + 2 * KVH) * D))
    cos = g.input("cos", (max_seq, D))
    sin = g.input("sin", (max_seq, D))
    pos = g.state("pos", (1, 1), torch.int32)
    kc = g.state("k_cache", (B * max_seq, KVH * D))
    vc = g.state("v_cache", (B * max_seq, KVH * D))
    q = g.rope_append(qkv, cos, sin, pos, kc, vc, heads=H, kv_heads=KVH, head_dim=D, max_seq=max_seq)
    a = g.decode_attention(q, kc, vc, pos, heads=H, kv_heads=KVH, head_dim=D, max_seq=max_seq)
    g.increment(pos)
    if fused:
        g.output(a)
    else:
        g.output(a, q)
    cs, sn = W.rope_tables(max_seq, D)
    cache = lambda s: (torch.cat([rnd((B, ctx, KVH * D), 1, s), torch.zeros(B, max_seq - ctx, KVH * D, dtype=BF)], 1)
                       .reshape(B * max_seq, KVH * D).contiguous())
    t = {"qkv": rnd((B, (H + 2 * KVH) * D), 1, 1), "cos": cs, "sin": sn,
         "pos": torch.full((1, 1), ctx, dtype=torch.int32), "k_cache": cache(2), "v_cache": cache(3)}
    before = {n: t[n].clone() for n in ("k_cache", "v_cache")}
    outs, ref, st, rst, prog = run_both(g, t, cuda, steps=2)
    kinds = [o.kind for o in prog.g.ops]
    assert ("RopeAppend" not in kinds) == fused
    assert_close(outs, ref)
    assert int(st["pos"]) == ctx + 2 == int(rst["pos"])
    for n in ("k_cache", "v_cache"):
        got, want = st[n].view(B, max_seq, -1), rst[n].view(B, max_seq, -1)
        old = before[n].view(B, max_seq, -1)
        # exactly rows ctx and ctx+1 of every sequence changed (integer-exact append slots)
        changed = (got != old).any(-1)
        mask = torch.zeros(B, max_seq, dtype=torch.bool)
        mask[:, ctx:ctx + 2] = True
        assert not changed[~mask].any()
        assert rel_l2(got[:, ctx:ctx + 2].float(), want[:, ctx:ctx + 2].float()) < TOL
    for b in prog.g.buffers:
        if b.kind == "workspace" and b.dtype == torch.int32:
            assert int(prog.buffer(b).abs().sum()) == 0
    assert np.array_equal(prog.counters(), prog.sched.counter_target * 2)
    return prog


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("B", [1, 2, 8])
def test_small_llama_decode_steps(cuda, B):
    g, params, st, ids = small_decode(B=B, E=256, H=4, KVH=2, F=512, n=3, max_seq=256, ctx=70, vocab=1000)
    prog = mc.compile(g)
    dp = {k: v.to(cuda) for k, v in params.items()}
    ds = {k: v.to(cuda) for k, v in st.items()}
    rs = {k: v.clone() for k, v in st.items()}
    emb = params["lm_head"]
    ids_g, ids_r = ids.clone(), ids.clone()
    for step in range(6):
        ds["x"].copy_(dp["lm_head"][ids_g.to(cuda)])
        logits = prog(**dp, **ds).float().cpu()
        rs["x"] = emb[ids_r].clone()
        ref, new = evaluate(g, {**params, **rs})
        for n in ("pos", "k_cache", "v_cache"):
            rs[n] = new[n]
        assert rel_l2(logits, ref[0]) < TOL, (step, rel_l2(logits, ref[0]))
        ids_g, ids_r = logits.argmax(-1), ref[0].argmax(-1)
        assert torch.equal(ids_g, ids_r)
        assert int(ds["pos"]) == int(rs["pos"]) == 71 + step
    prog.check()
    assert np.array_equal(prog.counters(), prog.sched.counter_target * 6)


def test_timeout_is_reported_not_hung(cuda):
    """Host-made fault: a wait target no arrival can satisfy.  The launch must end with an error
    status within the (shortened) limit and the program must be reusable after reset()."""
    g = mc.Graph()
    x = g.input("x", (1, 512))
    h = g.linear(x, g.param("w1", (512, 512)))
    g.output(g.linear(h, g.param("w2", (512, 512))))
    t = {"x": rnd((1, 512), 1, 1).to(cuda), "w1": rnd((512, 512), 0.04, 2).to(cuda), "w2": rnd((512, 512), 0.04, 3).to(cuda)}
    prog = mc.compile(g)
    good = prog(**t).float().cpu().clone()
    prog.check()
    from megacute_b200 import _lib
    prog.set_timeout(0.05)
    s = prog.sched
    _lib.check(_lib.load().mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), int(s.wait_tgt[0]) + 1000))
    prog(**t)
    with pytest.raises(_lib.MegakernelTimeout):
        prog.check()
    _lib.check(_lib.load().mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), int(s.wait_tgt[0])))
    prog.reset()
    again = prog(**t).float().cpu()
    prog.check()
    assert torch.equal(again, good)


@pytest.mark.parametrize("first", ["norm", "pointwise", "128-row tile", "256-row tile", "attention"])
def test_timeout_of_the_first_instruction(cuda, monkeypatch, first):
    """The very first instruction of the program waits for a counter that is never reached: CTA 0 leaves, although its body would
    have gone on with the CTA's next instructions, and the program works once the wait is put right."""
    from megacute_b200 import _lib, passes
    from megacute_b200.runtime import Program
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 128) if first == "256-row tile" else (1, 128, 128))
    M, N = 4096, 1024
    g = mc.Graph()
    x = g.input("x", (M, N))
    t = {"x": rnd((M, N), 1.0, 1)}
    if first == "norm":
        y = g.rms_norm(x)
    elif first == "pointwise":
        y = g.unary(x, "silu")
    elif first == "attention":
        y = g.attention(x, x, x, batch=8, heads=16, head_dim=64, causal=True)
    else:
        t["w"] = rnd((N, N), 0.03, 2)
        y = g.linear(x, g.param("w", (N, N)))
    g.output(g.unary(y, "neg"))
    prog = Program(g)
    s = prog.sched
    s.wait_ptr = s.wait_ptr.copy()
    s.wait_ptr[1:] += 1
    s.wait_cnt, s.wait_tgt = np.concatenate([[0], s.wait_cnt]), np.concatenate([[1000], s.wait_tgt])
    prog.compile()
    prog.set_timeout(0.05)
    dev = {k: v.to(cuda) for k, v in t.items()}
    prog(**dev)
    with pytest.raises(_lib.MegakernelTimeout):
        prog.check()
    _lib.check(_lib.load().mk_program_poke_wait(prog._handle, 0, 0, 0))
    prog.reset()
    prog.set_timeout(2.0)
    out = prog(**dev)
    prog.check()
    ref, _ = evaluate(g, t)
    assert rel_l2(out.float().cpu(), ref[0]) < TOL


def test_timeline(cuda):
    g, params, st, ids = small_decode(B=1, n=2)
    prog = mc.compile(g, trace=True)
    with pytest.raises(RuntimeError):
        mc.compile(g).timeline()
    dp = {k: v.to(cuda) for k, v in {**params, **st}.items()}
    prog(**dp)
    tl = prog.timeline()
    assert len([r for r in tl.records if r[1] == 1]) == prog.sched.n
    assert tl.span_us() > 0 and "Linear" in tl.summary() and len(tl.chrome_events()) > 0


def test_timeline_of_tile_gemm_runs(cuda):
    """A CTA that gets several tile-GEMM instructions in a row runs them inside one call of the body, which then writes
    the trace records itself: every instruction must still have exactly one record, under its own sequence number,
    with ordered time stamps and phase marks."""
    import numpy as np
    M, K = 4096, 512
    g = mc.Graph()
    x = g.input("x", (M, K))
    y = g.linear(g.unary(x, "identity"), g.param("w1", (1024, K)), act="gelu_tanh")     # 32 x 4 (or 8) tiles: 2 or more per CTA
    g.output(g.linear(y, g.param("w2", (384, 1024))))                                    # narrow tiles behind them
    gen = torch.Generator().manual_seed(5)
    t = {"x": torch.randn(M, K, generator=gen).to(torch.bfloat16), "w1": (torch.randn(1024, K, generator=gen) * 0.04).to(torch.bfloat16),
         "w2": (torch.randn(384, 1024, generator=gen) * 0.03).to(torch.bfloat16)}
    prog = mc.compile(g, trace=True)
    dp = {k: v.to(cuda) for k, v in t.items()}
    for _ in range(2):
        prog(**dp)
    prog.check()
    tl = prog.timeline()
    comp = tl.table[tl.table["role"] == 1]
    assert len(comp) == prog.sched.n and np.array_equal(np.sort(comp["seq"]), np.arange(prog.sched.n))
    assert bool((comp["t0"] <= comp["t1"]).all()) and bool((comp["t1"] < comp["t2"]).all())
    per_op = np.bincount(np.asarray(prog.sched.op_of)[comp["seq"]], minlength=len(prog.g.ops))
    assert np.array_equal(per_op, np.bincount(np.asarray(prog.sched.op_of), minlength=len(prog.g.ops)))
    # a CTA runs its instructions in list order: sequence numbers rise with the slot
    for sm in np.unique(comp["sm"])[:8]:
        rows = comp[comp["sm"] == sm]
        assert bool((np.diff(rows["seq"]) > 0).all()) and bool((np.diff(rows["t2"]) > 0).all())
    ph = tl.table[tl.table["role"] == 2]
    gemm = np.array([prog.g.ops[int(k)].kind in ("Linear", "LinearSplit") for k in np.asarray(prog.sched.op_of)[ph["seq"]]])
    by_seq = {int(r["seq"]): r for r in comp}
    for r in ph[gemm][:256]:
        c = by_seq[int(r["seq"])]
        assert c["t1"] <= r["t0"] <= r["t1"] <= r["t2"] <= c["t2"], (r, c)


# ---------------------------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 128256), (64, 128256), (3, 1000), (2, 8)])
def test_argmax_rows(cuda, dtype, rows, cols):
    g = torch.Generator(device=cuda).manual_seed(rows * 131 + cols)
    x = torch.randn(rows, cols, generator=g, device=cuda, dtype=torch.float32).to(dtype)
    # plant a unique maximum per row, and a tie whose lower index must win in row 0
    want = torch.randint(0, cols, (rows,), generator=g, device=cuda)
    x[torch.arange(rows, device=cuda), want] = 100.0
    if cols > 8:
        lo = int(want[0])
        hi = min(cols - 1, lo + 5)
        x[0, hi] = 100.0
    got = mc.argmax(x)
    assert got.dtype == torch.int64 and torch.equal(got, want)
    # a view with a leading dimension larger than its width
    wide = torch.zeros(rows, cols + 16, device=cuda, dtype=dtype)
    wide[:, :cols] = x
    assert torch.equal(mc.argmax(wide[:, :cols]), want)


def _chain(M, widths, residual_every=2):
    """Streaming linears one behind the other (direct operands: every hop by value), some with a residual from two hops before."""
    g = mc.Graph()
    x, t = g.input("x", (M, widths[0])), {"x": rnd((M, widths[0]), 1.0, 1)}
    hs = [x]
    for i, n in enumerate(widths[1:]):
        w = g.param(f"w{i}", (n, widths[i]))
        t[f"w{i}"] = rnd((n, widths[i]), widths[i] ** -0.5, 10 + i)
        res = hs[-2] if i % residual_every == 1 and hs[-2].shape == (M, n) else None
        hs.append(g.linear(hs[-1], w, residual=res))
    g.output(hs[-1])
    return g, t, hs


@pytest.mark.parametrize("M,widths", [(1, [256, 2048, 256, 2048, 256]), (2, [512, 2064, 512, 2064, 512, 16]), (8, [1040, 1024, 1040, 1024, 1040]),
                                      (5, [2048, 2048, 2048, 2048, 48, 2048]), (1, [8208, 48, 8208, 48])])
def test_values_instead_of_counters(cuda, M, widths):
    """Rows of one to many vectors per thread, K that is no multiple of 2048, fewer outputs than SMs, residuals by value; launch after launch
    with another input each, so that both copies of the buffers are used and filled again."""
    g, t, hs = _chain(M, widths)
    prog = mc.compile(g)
    assert len(prog.direct) == len(widths) - 2 and len(prog.sched.wait_cnt) == 0
    dev = {k: v.to(cuda) for k, v in t.items()}
    for step in range(5):
        dev["x"].copy_(rnd((M, widths[0]), 1.0, 50 + step))
        out = prog(**dev).float()
        ref, _ = evaluate(g, dev, cuda)
        prog.check()
        assert rel_l2(out, ref[0]) < TOL, step
        # the buffers hold this launch's values
        last = next(b for b in prog.g.buffers if b.id in prog.direct and b.name == hs[-2].buf.name)
        assert not bool((prog.buffer(last).view(torch.int32) == -1).any())


@pytest.mark.parametrize("by_value", [False, True])
@pytest.mark.parametrize("M,K", [(2, 256), (2, 8192), (3, 768), (5, 2048), (7, 2304), (8, 2048), (4, 2064), (8, 272)])
def test_rows_staged_side_by_side(cuda, monkeypatch, M, K, by_value):
    """Two rows and more of a private fp32 activation, K a multiple of 256 (two rows at a time; an odd last row alone) or not, with the
    norm's gain and sums of squares, rows of very different size.  One rounding of the result to bf16 is at most 2^-9; the
    operands' high and low parts leave 2^-16 of them."""
    monkeypatch.setattr(C, "DIRECT_MIN_COLS", 0 if by_value else 1 << 30)
    g = mc.Graph()
    h = g.linear(g.input("x", (M, 64)), g.param("v", (K, 64)))
    g.output(g.linear(g.rms_norm(h, g.param("n", (1, K)), eps=1e-5), g.param("w", (1000, K))))
    t = {"x": rnd((M, 64), 1.0, 1) * torch.tensor([4.0 ** (m % 5 - 2) for m in range(M)]).to(BF)[:, None], "v": rnd((K, 64), 0.1, 2),
         "n": rnd((1, K), 0.3, 3, 1.0), "w": rnd((1000, K), K ** -0.5, 4)}
    outs, ref, _, _, prog = run_both(g, t, cuda, steps=3)
    assert len(prog.direct) == (1 if by_value else 0)
    for r in range(M):
        assert rel_l2(outs[0][r], ref[0][r]) < 1.05 * 2.0 ** -9, r


@pytest.mark.parametrize("M", [1, 64])
@pytest.mark.parametrize("where", ["default stream", "side stream", "captured"])
def test_launches_behind_kernels_that_write_their_inputs(cuda, M, where):
    """A launch is prepared while the kernel in front of it runs: it must still see all of that one's writes -- input, weights, the output
    of the launch before -- and the kernel behind it all of its own."""
    K, N = 512, 512
    g = mc.Graph()
    g.output(g.linear(g.rms_norm(g.input("x", (M, K)), g.param("n", (1, K)), eps=1e-5), g.param("w", (N, K))))
    prog = mc.compile(g)
    xs = [rnd((M, K), 1.0, i).to(cuda) for i in range(8)]
    n, w = rnd((1, K), 0.1, 20, 1.0).to(cuda), rnd((N, K), K ** -0.5, 21).to(cuda)
    x, out, big = torch.zeros_like(xs[0]), torch.zeros((8, M, N), dtype=BF, device=cuda), torch.zeros(1 << 24, device=cuda)

    def steps():
        for i in range(8):
            big.add_(1.0)                        # (a kernel of all SMs whose last blocks end just before the next one)
            x.copy_(xs[i])
            y = prog(x=x, n=n, w=w)
            out[i].copy_(y)
            x.copy_(y)                           # the next launch's input is this one's output, overwritten
            y = prog(x=x, n=n, w=w)
            out[i].add_(y)

    want = []
    for i in range(8):
        y0 = prog(x=xs[i], n=n, w=w).clone()
        torch.cuda.synchronize()
        y1 = prog(x=y0, n=n, w=w).clone()
        torch.cuda.synchronize()
        want.append(y0 + y1)
    if where == "default stream":
        for _ in range(20):
            steps()
    else:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            steps()
        side.synchronize()
        out.zero_()
        if where == "side stream":
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                for _ in range(20):
                    steps()
            side.synchronize()
        else:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                steps()
            graph.replay()
    torch.cuda.synchronize()
    prog.check()
    for i in range(8):
        assert torch.equal(out[i], want[i]), i


@pytest.mark.parametrize("M", [1, 4, 64])
def test_replays_of_a_captured_launch(cuda, M):
    """A graph of one launch, replayed: each replay waits for its own values, in private buffers that hold no numbers and behind replays and
    launches with other inputs."""
    K = 4096 if M == 1 else 512                  # (one row: direct operands)
    g = mc.Graph()
    y = g.input("x", (M, K))
    for i in range(4):
        y = g.linear(g.rms_norm(y, g.param("n", (1, K)), eps=1e-5), g.param(f"w{i}", (K, K)), act="gelu_tanh")
    g.output(y)
    prog = mc.compile(g)
    t = {"n": rnd((1, K), 0.1, 20, 1.0).to(cuda), **{f"w{i}": rnd((K, K), 2 * K ** -0.5, 21 + i).to(cuda) for i in range(4)}}
    xs = [rnd((M, K), 1.0, i).to(cuda) for i in range(5)]
    x = torch.zeros_like(xs[0])
    want = [prog(x=v, **t).clone() for v in xs]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        prog(x=x, **t)
    side.synchronize()
    assert len(prog.direct) == (3 if M == 1 else len(prog.direct))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = prog(x=x, **t)
    private = [prog._bufs[b.id] for b in prog.g.buffers if b.kind == "temp" and b.id not in prog.direct]
    for k in (0, 1, 2, 3, 4, 1, 0):
        for b in private:
            b.fill_(float("nan"))
        x.copy_(xs[k])
        graph.replay()
        torch.cuda.synchronize()
        assert rel_l2(out.float().cpu(), want[k].float().cpu()) < TOL, k
        if k in (2, 4):                          # a launch of its own between replays
            x.copy_(xs[3])
            assert rel_l2(prog(x=x, **t).float().cpu(), want[3].float().cpu()) < TOL
    prog.check()


def test_values_that_are_nan_end_the_wait(cuda):
    """NaN inputs reach the output as NaN through direct operands; the rows beside them and the launches after are right.  (The input has
    all 16 bits set.  No op can produce the 32-bit marker itself: arithmetic makes 0x7fffffff, an embedding's low half is 0.)"""
    g, t, _ = _chain(2, [512, 2048, 512, 2048, 512])
    prog = mc.compile(g)
    dev = {k: v.to(cuda) for k, v in t.items()}
    clean = prog(**dev).clone()
    x = dev["x"].clone()
    dev["x"].view(torch.int16)[1, 100:104] = -1                      # bf16 0xffff
    out = prog(**dev)
    prog.check()
    assert torch.equal(out[0], clean[0]) and bool(out[1].isnan().all())
    dev["x"].copy_(x)
    for _ in range(2):
        assert torch.equal(prog(**dev), clean)


def test_values_that_never_come_end_the_launch(cuda):
    """A launch whose first op cannot start (a wait that cannot end) ends for the ops behind it too, which wait for values; the program gives
    the same result after a reset."""
    from megacute_b200 import _lib
    g = mc.Graph()
    x = g.input("x", (2, 512))
    t = {"x": rnd((2, 512), 1.0, 1)}
    h = g.unary(x, "silu")
    for i in range(4):
        t[f"w{i}"] = rnd((512, 512), 0.05, 2 + i)
        h = g.linear(h, g.param(f"w{i}", (512, 512)))
    g.output(h)
    prog = mc.compile(g)
    assert len(prog.direct) == 3 and len(prog.sched.wait_cnt) > 0
    dev = {k: v.to(cuda) for k, v in t.items()}
    want = prog(**dev).clone()
    prog.check()
    s = prog.sched
    prog.set_timeout(0.02)
    _lib.check(_lib.load().mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), 1000))
    prog(**dev)
    with pytest.raises(_lib.MegakernelTimeout):
        prog.check()
    _lib.check(_lib.load().mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), int(s.wait_tgt[0])))
    prog.reset()
    for _ in range(3):
        assert torch.equal(prog(**dev), want)
    prog.check()


def test_direct_operands_are_checked_at_bind_time(cuda):
    """A direct operand of a program without direct memory is refused as the descriptors are bound."""
    import ctypes
    from megacute_b200 import _lib
    g = mc.Graph()
    g.output(g.linear(g.input("x", (1, 256)), g.param("w", (256, 256))))
    t = {"x": rnd((1, 256), 1.0, 1).to(cuda), "w": rnd((256, 256), 0.05, 2).to(cuda)}
    prog = mc.compile(g)
    want = prog(**t).clone()
    lib = _lib.load()
    for flag in (8, 16, 32):
        prog._desc[0].flags |= flag
        assert lib.mk_program_set_ops(prog._handle, ctypes.addressof(prog._desc), 1, None) == -2
        assert b"direct operands" in lib.mk_last_cuda_error()
        prog._desc[0].flags &= ~flag
    assert torch.equal(prog(**t), want)


def _gated_decode(B=2, H=8, KVH=2, D=64, L=128, ctx=40):
    """pointwise op (behind counters) -> QKV -> decode attention -> O: every hop behind the first linear by value."""
    E = 512
    g = mc.Graph()
    x = g.input("x", (B, E))
    t = {"x": rnd((B, E), 1.0, 1), "wqkv": rnd(((H + 2 * KVH) * D, E), E ** -0.5, 2), "wo": rnd((512, H * D), (H * D) ** -0.5, 3),
         "pos": torch.full((1, 1), ctx, dtype=torch.int32)}
    t["cos"], t["sin"] = W.rope_tables(L, D)
    for i, n in enumerate(("k_cache", "v_cache")):
        t[n] = rnd((B * L, KVH * D), 1.0, 4 + i)
    cos, sin, pos = g.input("cos", (L, D)), g.input("sin", (L, D)), g.state("pos", (1, 1), torch.int32)
    kc, vc = (g.state(n, (B * L, KVH * D)) for n in ("k_cache", "v_cache"))
    qkv = g.linear(g.unary(x, "silu"), g.param("wqkv", t["wqkv"].shape))
    q = g.rope_append(qkv, cos, sin, pos, kc, vc, heads=H, kv_heads=KVH, head_dim=D, max_seq=L)
    a = g.decode_attention(q, kc, vc, pos, heads=H, kv_heads=KVH, head_dim=D, max_seq=L)
    h = g.linear(a, g.param("wo", t["wo"].shape))
    t["w2"], t["w3"] = rnd((512, 512), 0.04, 6), rnd((512, 512), 0.04, 7)
    g.output(g.linear(g.linear(h, g.param("w2", (512, 512))), g.param("w3", (512, 512)), residual=h))
    return g, t


def test_wait_for_values_that_ends_leaves_the_callers_tensors_alone(cuda):
    """The values an attention and the linears behind it wait for never come: the launch ends with the status of a dependency that was not
    met, nothing made without them is written to the caller's cache and output, and the step after a reset is right."""
    from megacute_b200 import _lib
    g, t = _gated_decode()
    prog = mc.compile(g)
    assert len(prog.direct) == 4 and len(prog.sched.wait_cnt) > 0
    dev = {k: v.to(cuda) for k, v in t.items()}
    s, lib = prog.sched, _lib.load()
    out = prog(**dev)
    prog.check()
    ref, st = evaluate(g, t)
    for _ in range(3):
        for k in ("k_cache", "v_cache", "pos"):
            dev[k].copy_(t[k])
        out.zero_()
        prog.set_timeout(0.02)
        _lib.check(lib.mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), 1000))
        prog(**dev)
        with pytest.raises(_lib.MegakernelTimeout, match="dependency"):
            prog.check()
        # the linear that is stuck makes q of the first kv head; other heads may have appended their rows, with their values
        for k in ("k_cache", "v_cache"):
            got = dev[k].cpu().float()
            assert torch.equal(got[:, :64], t[k][:, :64].float())
            changed = got != t[k].float()
            assert rel_l2(torch.where(changed, got, st[k].float()), st[k].float()) < TOL
        assert not out.any()
        _lib.check(lib.mk_program_poke_wait(prog._handle, 0, int(s.wait_cnt[0]), int(s.wait_tgt[0])))
        prog.reset()
        prog.set_timeout(2.0)
        got = prog(**dev).float().cpu()
        prog.check()
        assert rel_l2(got, ref[0]) < TOL and rel_l2(dev["k_cache"].cpu().float(), st["k_cache"].float()) < TOL


@pytest.mark.parametrize("H,KVH,D,B,ctx", [(8, 2, 128, 2, 40), (8, 1, 128, 1, 200), (8, 1, 64, 3, 40), (4, 4, 128, 8, 0), (16, 2, 64, 1, 127)])
def test_decode_attention_by_value(cuda, H, KVH, D, B, ctx):
    """Direct q, k, v and output of the decode attention at both head sizes and groups of 1, 4 and 8, launch after launch with another input."""
    L = 256
    g, t = _gated_decode(B, H, KVH, D, L, ctx)
    prog = mc.compile(g)
    att = next(o for o in prog.g.ops if o.kind == "DecodeAttention")
    assert {att.q.buf.id, att.out.buf.id} <= prog.direct and att.k_new is not None
    dev, ref_t = {k: v.to(cuda) for k, v in t.items()}, dict(t)
    for step in range(4):
        ref_t["x"] = rnd((B, 512), 1.0, 30 + step)
        dev["x"].copy_(ref_t["x"])
        got = prog(**dev).float().cpu()
        prog.check()
        ref, st = evaluate(g, ref_t)
        assert rel_l2(got, ref[0]) < TOL, step
        for n in ("k_cache", "v_cache"):
            ref_t[n] = st[n]
            assert rel_l2(dev[n].cpu().float(), st[n].float()) < TOL, (step, n)


@pytest.mark.parametrize("splits", [1, 2, 3, 5])
def test_many_sequence_attention_with_infinite_values(cuda, monkeypatch, splits):
    """Infinite elements of the new token's v reach the output as they are, whatever the number of splits (the last one merges them in pairs)."""
    monkeypatch.setenv("MEGACUTE_B200_ATT_BULK", "1")
    monkeypatch.setenv("MEGACUTE_B200_KV_SPLITS", str(splits))
    B, H, KVH, D, L, ctx = 12, 16, 4, 64, 1024, 960                   # (whole tiles in every split)
    g = mc.Graph()
    x = rnd((B, (H + 2 * KVH) * D), 1.0, 1)
    x[:, (H + KVH) * D + 5], x[:, (H + KVH) * D + 6] = float("inf"), -float("inf")
    t = {"qkv": x, "pos": torch.full((1, 1), ctx, dtype=torch.int32), "k_cache": rnd((B * L, KVH * D), 1.0, 2), "v_cache": rnd((B * L, KVH * D), 1.0, 3)}
    t["cos"], t["sin"] = W.rope_tables(L, D)
    pos, kc, vc = g.state("pos", (1, 1), torch.int32), g.state("k_cache", (B * L, KVH * D)), g.state("v_cache", (B * L, KVH * D))
    q = g.rope_append(g.input("qkv", x.shape), g.input("cos", (L, D)), g.input("sin", (L, D)), pos, kc, vc, heads=H, kv_heads=KVH, head_dim=D, max_seq=L)
    g.output(g.decode_attention(q, kc, vc, pos, heads=H, kv_heads=KVH, head_dim=D, max_seq=L))
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert all(o.bulk and o.splits == splits for o in prog.g.ops if o.kind == "DecodeAttention")
    got, ref = outs[0].view(B, H, D), ref[0].view(B, H, D)
    assert torch.equal(got.isinf(), ref.isinf()) and torch.equal(got.sign()[got.isinf()], ref.sign()[ref.isinf()])
    fin = ~ref.isinf()
    assert int(ref.isinf().sum()) == 2 * B * H // KVH and rel_l2(got[fin], ref[fin]) < TOL


@pytest.mark.parametrize("ctx", [0, 1, 15, 16, 37, 301])
@pytest.mark.parametrize("form", ["per head", "many sequences"])
def test_cache_rows_that_nothing_has_written_yet(cuda, monkeypatch, form, ctx):
    """Rows at and behind the position hold NaN (memory that was never written): no output depends on them."""
    monkeypatch.setenv("MEGACUTE_B200_ATT_BULK", str(int(form != "per head")))
    monkeypatch.setenv("MEGACUTE_B200_KV_SPLITS", "2")
    B, H, KVH, D, L = 9, 16, 4, 64, 384
    g = mc.Graph()
    t = {"qkv": rnd((B, (H + 2 * KVH) * D), 1.0, 1), "pos": torch.full((1, 1), ctx, dtype=torch.int32)}
    t["cos"], t["sin"] = W.rope_tables(L, D)
    for i, n in enumerate(("k_cache", "v_cache")):
        t[n] = rnd((B * L, KVH * D), 1.0, 2 + i)
        t[n].view(B, L, -1)[:, ctx:] = float("nan")
    pos, kc, vc = g.state("pos", (1, 1), torch.int32), g.state("k_cache", (B * L, KVH * D)), g.state("v_cache", (B * L, KVH * D))
    q = g.rope_append(g.input("qkv", t["qkv"].shape), g.input("cos", (L, D)), g.input("sin", (L, D)), pos, kc, vc, heads=H, kv_heads=KVH, head_dim=D, max_seq=L)
    g.output(g.decode_attention(q, kc, vc, pos, heads=H, kv_heads=KVH, head_dim=D, max_seq=L))
    outs, ref, _, _, prog = run_both(g, t, cuda)
    assert all(bool(o.bulk) == (form != "per head") for o in prog.g.ops if o.kind == "DecodeAttention")
    assert_close(outs, ref)


def test_timeline_shows_waits_for_values(cuda):
    """The wait of an instruction with a direct operand lasts until the values are there: most SMs have no part in a linear of 48 outputs and
    wait for the next one's input for as long as it takes."""
    g, t, _ = _chain(1, [2048, 2048, 48, 2048, 48, 2048])
    prog = mc.compile(g, trace=True)
    dev = {k: v.to(cuda) for k, v in t.items()}
    for _ in range(3):
        prog(**dev)
    prog.check()
    comp = prog.timeline().table
    comp = comp[comp["role"] == 1]
    assert bool((comp["t0"] <= comp["t1"]).all()) and bool((comp["t1"] <= comp["t2"]).all())
    op = np.asarray(prog.sched.op_of)[comp["seq"]]
    for k in (2, 4):
        assert prog.g.ops[k].x.cols == 48 and prog.g.ops[k].x.buf.id in prog.direct
        assert np.median((comp["t1"] - comp["t0"])[op == k]) > 500                   # (ns; a linear takes 1.5 us at least)


def test_direct_operands_must_lie_in_their_memory(cuda):
    """A program with direct memory: each thing its kernel relies on changed by itself is refused as the descriptors are bound -- type,
    path, an operand that starts outside or runs past the end of the first copy, a misaligned one -- and the program still runs."""
    import ctypes
    from megacute_b200 import _lib
    from megacute_b200 import config as C
    g, t = _gated_decode()
    prog = mc.compile(g)
    dev = {k: v.to(cuda) for k, v in t.items()}
    want = prog(**dev).clone()
    prog.check()
    lib, n = _lib.load(), len(prog.g.ops)
    ops = {o.kind: k for k, o in enumerate(prog.g.ops)}
    att = ops["DecodeAttention"]
    lin = next(k for k, o in enumerate(prog.g.ops) if o.kind == "Linear" and prog._desc[k].flags & C.F_DIRECT_RES)
    base, size = prog._direct_mem.data_ptr(), prog._direct_mem.shape[1] * 4
    refused = []

    def change(k, field, index, value):
        d = prog._desc[k]
        seq = getattr(d, field) if index is not None else None
        old = seq[index] if index is not None else getattr(d, field)
        new = value(old)
        if index is not None:
            seq[index] = new
        else:
            setattr(d, field, new)
        rc = lib.mk_program_set_ops(prog._handle, ctypes.addressof(prog._desc), n, None)
        refused.append((k, field, index))
        assert rc == -2 and b"direct operands" in lib.mk_last_cuda_error(), refused[-1]
        if index is not None:
            seq[index] = old
        else:
            setattr(d, field, old)

    for at, dt in ((0, 4), (4, 6)):                                           # a linear's x and residual
        change(lin, "i", dt, lambda v: 0)                                     # another type
        change(lin, "ptr", at, lambda v: base - 16)                           # before the memory
        change(lin, "ptr", at, lambda v: base + size)                         # behind the first copy
        change(lin, "ptr", at, lambda v: base + size - 16)                    # past its end
        change(lin, "ld", at, lambda v: size // 4)                            # ... with its second row
    change(lin, "ptr", 0, lambda v: v + 4)                                    # 16-byte loads
    change(lin, "ld", 0, lambda v: v + 1)
    change(lin, "flags", None, lambda v: v & ~4)                              # not the tensor-core path
    for at in (0, 5, 6, 4):                                                   # the attention's q, k, v and output
        change(att, "ptr", at, lambda v: base + size - 16)
    change(att, "i", 7, lambda v: 0)
    change(att, "i", 8, lambda v: 0)
    change(att, "i", 9, lambda v: 1)                                          # inputs zeroed behind the read
    change(att, "i", 6, lambda v: 0)                                          # not fused
    assert lib.mk_program_set_ops(prog._handle, ctypes.addressof(prog._desc), n, None) == 0
    for k in ("k_cache", "v_cache", "pos"):
        dev[k].copy_(t[k])
    assert torch.equal(prog(**dev), want)
    prog.check()


def test_timeout_in_a_step_with_several_heads_per_instruction(cuda, monkeypatch):
    """A wait that cannot end, at the first waiting instruction of every op of a batched decode step whose attention instructions run
    several kv heads each: the launch ends, and the step is right once the wait is."""
    from megacute_b200 import _lib
    monkeypatch.setenv("MEGACUTE_B200_ATT_HEADS", "2")
    monkeypatch.setenv("MEGACUTE_B200_ATT_BULK", "0")
    g, params, st, _ = small_decode(B=16, E=256, H=4, KVH=2, F=512, n=1, max_seq=256, ctx=120, vocab=1000)
    prog = mc.compile(g)
    assert {o.heads_per_inst for o in prog.g.ops if o.kind == "DecodeAttention"} == {2}
    dp, ds = ({k: v.to(cuda) for k, v in d.items()} for d in (params, st))
    ref, _ = evaluate(g, {**params, **st})
    prog(**dp, **ds)
    prog.check()
    s, lib = prog.sched, _lib.load()
    prog.set_timeout(0.02)
    for k, (i0, i1) in enumerate(s.node_ranges):
        i = next((i for i in range(i0, i1) if s.wait_ptr[i + 1] > s.wait_ptr[i]), None)
        if i is None:
            continue
        at = int(s.wait_ptr[i])
        _lib.check(lib.mk_program_poke_wait(prog._handle, at, int(s.wait_cnt[at]), 1000))
        prog(**dp, **ds)
        with pytest.raises(_lib.MegakernelTimeout):
            prog.check()
        _lib.check(lib.mk_program_poke_wait(prog._handle, at, int(s.wait_cnt[at]), int(s.wait_tgt[at])))
        prog.reset()
        for n, v in st.items():
            ds[n].copy_(v)
        out = prog(**dp, **ds)
        prog.check()
        assert rel_l2(out.float().cpu(), ref[0]) < TOL, prog.g.ops[k].kind
