"""What the graph rewrites must refuse: graphs that look like the fused pattern and are not.  The rewritten graph has to
evaluate to what the graph says, in the oracle, which runs ops one after the other and rejects a read of a tensor that nothing wrote."""
import pytest
import torch

import megacute_b200 as mc
from megacute_b200 import encode, passes
from megacute_b200.schedule import schedule
from megacute_b200.verify import VerifyError, check_hazards, check_tables
from oracle.graph_oracle import evaluate, rel_l2

BF = torch.bfloat16
SMS = 148


def rnd(shape, std=1.0, seed=0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(BF)


def check_rewritten(g, tensors, tol=1e-5):
    """run_all(g) agrees with g (fp32 on both sides: sums in another order at most).  Returns its op kinds."""
    want, _ = evaluate(g, tensors)
    out = passes.run_all(g, SMS)
    got, _ = evaluate(out, tensors)
    for a, b in zip(got, want):
        assert rel_l2(a, b) < tol
    return [o.kind for o in out.ops]


@pytest.mark.parametrize("form", ["residual first", "gated first", "gate is the product"])
def test_gated_residual_of_the_product_itself(monkeypatch, form):
    """y + y * gate with y = linear(x): the linear of 256-row tiles still has to write y."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256))
    g = mc.Graph()
    x, w = g.input("x", (384, 64)), g.param("w", (256, 64))
    y = g.linear(x, w)
    t = {"x": rnd((384, 64)), "w": rnd((256, 64), 0.1, 1)}
    if form == "gate is the product":
        r = g.input("r", (384, 256))
        t["r"] = rnd((384, 256), 1.0, 2)
        g.output(g.add(r, g.binary(y, y.rows_slice(0, 192), "mul", b_group=2)))
    else:
        z = g.binary(y, g.input("gate", (6, 256)), "mul", b_group=64)
        t["gate"] = rnd((6, 256), 1.0, 2)
        g.output(g.add(y, z) if form == "residual first" else g.add(z, y))
    assert check_rewritten(g, t) == ["Linear", "Binary"]


@pytest.mark.parametrize("M,N", [(8, 64), (9, 64), (64, 136), (128, 64), (129, 256), (384, 128)])
@pytest.mark.parametrize("group", [2, 3, 32])
@pytest.mark.parametrize("gate_dtype", [BF, torch.float32])
@pytest.mark.parametrize("act", [None, "gelu_tanh", "swiglu"])
@pytest.mark.parametrize("splits", [1, 2])
def test_gated_residual_in_the_linear(monkeypatch, M, N, group, gate_dtype, act, splits):
    """Which linears take a gated residual: tile linears (more than eight rows), 128-row tiles with a 16-bit gate, no swiglu; and the
    SplitFinalize behind K splits, with any gate."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (min(splits, a[4]), 256, 128) if a[1] % 128 == 0 else (min(splits, a[4]), 128, 128))
    monkeypatch.setattr(passes, "choose_k_splits", lambda *a: splits)
    M = -(-M // group) * group
    g = mc.Graph()
    n = N // 2 if act == "swiglu" else N
    t = {"x": rnd((M, 64)), "w": rnd((N, 64), 0.1, 1), "r": rnd((M, n), 1.0, 2), "gate": rnd((M // group, n), 1.0, 3).to(gate_dtype)}
    if act == "swiglu" and N % 128:
        return
    y = g.linear(g.input("x", (M, 64)), g.param("w", (N, 64)), act=act)
    g.output(g.add(g.input("r", (M, n)), g.binary(y, g.input("gate", (M // group, n), gate_dtype), "mul", b_group=group)))
    wide = M > 128 and N % 128 == 0
    fused = act != "swiglu" and M > 8 and (wide or gate_dtype != torch.float32)
    if splits == 2 and act != "swiglu" and M > 8:
        assert check_rewritten(g, t) == ["LinearSplit", "SplitFinalize"]
    else:
        assert check_rewritten(g, t) == (["Linear"] if fused else ["Linear", "Binary"])


def rotated(g, S, H=2, KVH=1, D=64, tables=lambda c, s: (c, s), qkv_dtype=None):
    """x -> q, k, v of one prompt -> rotated q and k -> attention.  `tables`: ops between the linear and the rotation."""
    x, w = g.input("x", (S, 64)), g.param("w", ((H + 2 * KVH) * D, 64))
    c, s = g.input("cos", (S, D)), g.input("sin", (S, D))
    qkv = g.linear(x, w, out=g.temp((S, w.rows), dtype=qkv_dtype))
    c, s = tables(c, s)
    q = g.rope(qkv.cols_slice(0, H * D), c, s, heads=H, head_dim=D, seq=S)
    k = g.rope(qkv.cols_slice(H * D, KVH * D), c, s, heads=KVH, head_dim=D, seq=S)
    v = qkv.cols_slice((H + KVH) * D, KVH * D)
    if qkv_dtype:
        v = g.unary(v, "identity")
    g.output(g.attention(q, k, v, batch=1, heads=H, kv_heads=KVH, head_dim=D, causal=True))
    return {"x": rnd((S, 64)), "w": rnd((w.rows, 64), 0.1, 1), "cos": rnd((S, D), 1.0, 2), "sin": rnd((S, D), 1.0, 3)}


def test_rotation_stays_behind_the_op_that_makes_its_tables():
    g = mc.Graph()
    t = rotated(g, 80)
    assert check_rewritten(g, t) == ["Linear", "Attention"]
    for which in (0, 1):
        g = mc.Graph()
        t = rotated(g, 80, tables=lambda c, s: (g.unary(c, "neg"), s) if which == 0 else (c, g.unary(s, "neg")))
        assert check_rewritten(g, t) == ["Linear", "Unary", "Rope", "Rope", "Attention"]


def test_rotation_of_an_fp32_product_keeps_its_op():
    """q and k computed in fp32 and rotated into 16 bits: attention cannot read the fp32 buffer."""
    g = mc.Graph()
    t = rotated(g, 80, qkv_dtype=torch.float32)
    assert "Rope" in check_rewritten(g, t)
    for op in passes.run_all(g, SMS).ops:
        encode.validate(op)


@pytest.mark.parametrize("rows", [16, 64, 300])
def test_k_splits_do_not_add_into_their_own_input(rows):
    """h + linear(h): the splits of one tile must not be added into rows of h that another tile still reads."""
    g = mc.Graph()
    h = g.unary(g.input("x", (rows, 2048)), "relu")
    g.output(g.unary(g.linear(h, g.param("w", (2048, 2048)), residual=h), "identity"))
    split = [o for o in passes.run_all(g, SMS).ops if o.kind == "LinearSplit"]
    assert (split or rows > 128) and all(o.ws.buf is not v.buf for o in split for v in o.reads)


@pytest.mark.parametrize("form", ["read again", "overwritten"])
def test_k_splits_are_not_added_into_a_residual_that_lives_on(form):
    """Two linears add to the residual stream one after the other; the value in between is read (or the first one's memory is used
    for something else) afterwards."""
    g = mc.Graph()
    x, w, w2 = g.input("x", (16, 2048)), g.param("w", (2048, 2048)), g.param("w2", (2048, 2048))
    r = g.unary(x, "relu")
    y1 = g.linear(x, w, residual=r)
    if form == "read again":
        g.output(g.add(y1, g.linear(x, w2, residual=y1)))
    else:
        g.unary(x, "silu", out=r)
        g.output(g.unary(y1, "identity"))
    kinds = check_rewritten(g, {"x": rnd((16, 2048)), "w": rnd((2048, 2048), 0.02, 1), "w2": rnd((2048, 2048), 0.02, 2)})
    assert "SplitFinalize" in kinds


def test_pointwise_pairs_whose_middle_is_read_twice():
    """z + z with z = y * gate, and a norm modulated by itself: the op in the middle has to run."""
    g = mc.Graph()
    z = g.mul(g.input("a", (64, 64)), g.input("b", (4, 64)))
    g.output(g.add(z, z))
    assert check_rewritten(g, {"a": rnd((64, 64)), "b": rnd((4, 64), 1.0, 1)}) == ["Binary", "Binary"]
    g = mc.Graph()
    n, s = g.rms_norm(g.input("a", (64, 64))), g.input("s", (64, 64))
    g.output(g.modulate(g.modulate(n, n, s, group=1), s, s, group=1))
    assert check_rewritten(g, {"a": rnd((64, 64)), "s": rnd((64, 64), 1.0, 1)}) == ["Norm", "Modulate", "Modulate"]


def test_fused_ops_do_not_overwrite_what_they_read():
    """Graphs that put the second op's result where the first one's operands are.  Op by op they are right; in one op an instruction
    would write what another still reads."""
    def kinds(build):
        g = mc.Graph()
        build(g)
        return [o.kind for o in passes.run_all(g, SMS).ops]

    def norm_linear_in_place(g):                    # x = x + linear(rms_norm(x))
        x = g.state("x", (2, 256))
        g.linear(g.rms_norm(x), g.param("w", (256, 256)), residual=x, out=x)

    def modulate_shifted(g):                        # the rows one further
        x, s = g.state("x", (65, 64)), g.input("s", (1, 64))
        g.modulate(g.rms_norm(x.rows_slice(0, 64)), s, s, group=64, out=x.rows_slice(1, 64))

    def modulate_in_place(g):
        x, s = g.state("x", (64, 64)), g.input("s", (1, 64))
        g.modulate(g.rms_norm(x), s, s, group=64, out=x)

    def gated_over_its_gate(g):
        x = g.state("x", (64, 64))
        g.add(g.input("r", (64, 64)), g.binary(g.input("y", (64, 64)), x.rows_slice(0, 4), "mul", b_group=16), out=x)

    def attention_over_qkv(g):
        qkv, pos = g.state("qkv", (1, 256)), g.state("pos", (1, 1), torch.int32)
        c, s, k, v = g.input("c", (128, 64)), g.input("s", (128, 64)), g.state("k", (128, 64)), g.state("v", (128, 64))
        q = g.rope_append(qkv, c, s, pos, k, v, heads=2, kv_heads=1, head_dim=64, max_seq=128)
        g.decode_attention(q, k, v, pos, heads=2, kv_heads=1, head_dim=64, max_seq=128, out=qkv.cols_slice(64, 128))

    assert kinds(norm_linear_in_place) == ["Norm", "Linear"]
    assert kinds(modulate_shifted) == ["Norm", "Modulate"] and kinds(modulate_in_place) == ["Norm"]
    assert kinds(gated_over_its_gate) == ["Binary", "Binary"]
    assert kinds(attention_over_qkv) == ["RopeAppend", "DecodeAttention"]


def test_gated_residual_over_the_weights(monkeypatch):
    """The linear's other row tiles still read what the gated residual is put over."""
    monkeypatch.setattr(passes, "plan_tiles", lambda *a: (1, 256, 256))
    g = mc.Graph()
    w = g.state("w", (512, 256))
    y = g.linear(g.input("x", (512, 256)), w.rows_slice(0, 256))
    g.add(g.input("r", (512, 256)), g.binary(y, g.input("gate", (8, 256)), "mul", b_group=64), out=w)
    assert [o.kind for o in passes.run_all(g, SMS).ops] == ["Linear", "Binary"]


def test_verifier_rejects_reads_of_temps_nothing_wrote():
    g = mc.Graph()
    y = g.unary(g.input("x", (64, 64)), "relu")
    g.output(g.add(y, y))
    check_tables(g, schedule(g, SMS))
    bad = g.derive()
    bad.ops = bad.ops[1:]
    with pytest.raises(VerifyError, match="no earlier op writes"):
        check_tables(bad, schedule(bad, SMS))
    # a K split added into a residual that was never made
    g = mc.Graph()
    r = g.unary(g.input("x", (16, 2048)), "relu")
    g.output(g.unary(g.linear(g.input("h", (16, 2048)), g.param("w", (2048, 2048)), residual=r), "identity"))
    out = passes.run_all(g, SMS)
    assert "SplitFinalize" not in [o.kind for o in out.ops]
    check_tables(out, schedule(out, SMS))
    out.ops = [o for o in out.ops if o.kind != "Unary" or o.x.buf.kind == "temp"]
    with pytest.raises(VerifyError, match="no earlier op writes"):
        check_tables(out, schedule(out, SMS))


def test_verifier_rejects_an_op_that_overwrites_its_own_operand():
    """Instructions of one op run side by side: element by element in place is right, a linear over its own input is not."""
    g = mc.Graph()
    x = g.state("x", (300, 256))
    g.unary(x, "relu", out=x)
    check_hazards(schedule(g, SMS), g)
    g.linear(x, g.param("w", (256, 256)), out=x)
    with pytest.raises(VerifyError, match="with nothing between them"):
        check_hazards(schedule(g, SMS), g)


def test_direct_buffers_and_their_schedule():
    """Which buffers need no counters, and that the tables without them still order every hazard (the values' own order counted)."""
    from megacute_b200.builders import llama_decode, mlp_block
    from megacute_b200.passes import direct_buffers, run_all
    for B, ragged, per_layer in ((1, False, 5), (2, True, 5), (5, True, 2), (16, False, 0)):        # (5 rows: the down projection is a K split)
        g = run_all(llama_decode(B, 2048, 32, 8, 8192, 2, 256, 4096, 1e-5, ragged=ragged), 148)
        direct = direct_buffers(g)
        assert len(direct) == 2 * per_layer
        s, plain = schedule(g, 148, direct), schedule(g, 148)
        check_tables(g, s)
        assert check_hazards(s, g) == check_hazards(plain, g)
        assert bool(s.value_deps) == bool(direct) and (len(s.wait_cnt) < len(plain.wait_cnt)) == bool(direct)
        if direct:                                      # without the values' order the same tables are refused
            s.value_deps = {}
            with pytest.raises(VerifyError):
                check_hazards(s, g)
    assert len(direct_buffers(run_all(mlp_block(1, 2048, 5632), 148))) == 1
    assert not direct_buffers(run_all(mlp_block(1, 512, 512), 148))                                 # (a narrow hop alone)
    # read by an op that cannot wait for values; visible to the caller; read in 16 bits; written in part
    for case in ("unary", "output", "rows", "part"):
        g = mc.Graph()
        x, w = g.input("x", (16 if case == "rows" else 1, 2048)), g.param("w", (4096, 2048))
        v = g.param("v", (2048, 4096))
        if case == "part":
            h = g.temp((1, 8192))
            g.linear(x, w, out=h.cols_slice(0, 4096))
            g.linear(x, w, out=h.cols_slice(4096, 4096))
            g.output(g.linear(h.cols_slice(0, 4096), v))
        else:
            h = g.linear(x, w)
            g.output(g.linear(h, v))
            if case == "unary":
                g.output(g.unary(h, "relu"))
            if case == "output":
                g.output(h)
        assert not direct_buffers(run_all(g, 148)), case


def test_few_narrow_hops_keep_their_counters():
    """One or two direct buffers pay from config.DIRECT_MIN_COLS columns on, three or more at any width."""
    from megacute_b200 import config as C
    from megacute_b200.passes import direct_buffers, run_all

    def direct(*widths):
        g = mc.Graph()
        h = g.input("x", (1, widths[0]))
        for i, n in enumerate(widths[1:]):
            h = g.linear(h, g.param(f"w{i}", (n, h.cols)))
        g.output(h)
        return len(direct_buffers(run_all(g, SMS)))

    wide = C.DIRECT_MIN_COLS
    assert direct(512, wide - 16, 512) == 0 and direct(512, wide, 512) == 1
    assert direct(512, wide - 16, wide - 16, 512) == 0 and direct(512, 64, wide, 512) == 2
    assert direct(512, 64, 64, 64, 512) == 3


def test_values_order_nothing_but_themselves():
    """A linear that reads a pointwise op's result beside a direct operand made from it needs its counter: the values it waits for were
    loaded and stored without an order for other accesses."""
    from megacute_b200.passes import run_all
    g = mc.Graph()
    u = g.unary(g.input("x", (1, 512)), "silu")
    h = g.linear(u, g.param("w1", (48, 512)))                # three instructions: most SMs have not waited for u before the second linear
    g.output(g.linear(h, g.param("w2", (512, 48)), residual=u))
    g = run_all(g, SMS)
    h = g.ops[1].out.buf.id
    assert [o.kind for o in g.ops] == ["Unary", "Linear", "Linear"]
    s = schedule(g, SMS, {h})
    check_hazards(s, g)
    b0 = s.node_ranges[2][0]
    at = int(s.wait_ptr[b0])
    assert at < len(s.wait_cnt) and all(buf == h for i in s.value_deps for buf, _ in s.value_deps[i])
    s.wait_ptr[b0:], s.wait_cnt, s.wait_tgt = at, s.wait_cnt[:at], s.wait_tgt[:at]
    with pytest.raises(VerifyError, match="unordered hazard"):
        check_hazards(s, g)
