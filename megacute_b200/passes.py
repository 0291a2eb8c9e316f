"""Graph rewrites applied by ``compile`` before scheduling: Graph -> Graph, each on a derived copy.

Same pass names and intent as the reference (``megacute/runtime.py:44-199``), re-decided for this
runtime's kernel:

  fold_norms           few-row RMSNorm feeding only linears -> computed inside those linears.
                       The reference folds the gain into a derived copy of the weights and applies
                       rstd in the GEMM epilogue; here the consuming instruction normalises its own
                       copy of the (<= 8 row) activation in shared memory before streaming weights,
                       so no second copy of any weight (e.g. the 525 MB lm_head) is made.
  split_k              tile GEMMs that cannot fill the SMs are split along K into partial
                       instructions that reduce-add into an fp32 workspace (+ SplitFinalize) or, for
                       a residual linear, straight into the residual stream.
  fuse_rope_attention  RopeAppend feeding only the next DecodeAttention -> one fused op.
  split_kv             decode attention instructions are multiplied along the key axis so that every
                       SM streams keys; the last split of a (sequence, kv head) pair to finish
                       combines the partials inside the op.
  fuse_gated_linear, fuse_rope_linear   gated residuals and the rotation of q and k into the epilogue of the
                       tile linear before them.
  hoist_linears        linears whose operands are ready long before their place move up.
  halve_last_tiles     the last rows of a long linear of few 256 x 256 tiles in tiles half as wide.
"""

from __future__ import annotations

import functools
import os

import torch

from . import config as C
from .graph import Buffer, Graph, Op, View


def _reads_buffer(ops, buf, outputs=()) -> bool:
    return any(v.buf is buf for op in ops for v in op.reads) or any(v.buf is buf for v in outputs)


def _overwrites(op, views, in_place=None) -> bool:
    """Does op write a buffer that one of `views` -- operands an op fused with it would read in all its instructions -- lies in?
    `in_place`: one more operand, that the fused op reads and writes element by element or row by row: it may be what op writes."""
    clash = lambda w, v: v is not None and w.buf is v.buf
    return any(clash(w, v) for w in op.writes for v in views) or any(clash(w, in_place) and not w.same(in_place) for w in op.writes)


def gemv_eligible(M: int, K: int) -> bool:
    """Does a linear with M activation rows of length K run on the weight-streaming GEMV path?
    The whole activation is kept in shared memory as fp32."""
    return M <= C.GEMV_MAX_ROWS and M * K * 4 <= C.GEMV_XBUF_BYTES


def fold_norms(g: Graph) -> Graph:
    out = g.derive()
    ops = list(g.ops)
    drop = set()
    for i, op in enumerate(ops):
        if not (op.kind == "Norm" and op.rms and op.bias is None and op.out.buf.kind == "temp"):
            continue
        if not gemv_eligible(op.x.rows, op.x.cols):
            continue
        users = [j for j in range(i + 1, len(ops)) if any(v.buf is op.out.buf for v in ops[j].reads)]
        ok = bool(users) and not _reads_buffer((), op.out.buf, g.outputs)
        for j in users:
            u = ops[j]
            ok = ok and u.kind == "Linear" and op.out.same(u.x) and u.rms_eps is None
            ok = ok and all(v is None or v.buf is not op.out.buf for v in (u.residual, u.bias))
        # the raw input must not be rewritten between the norm and its last user, nor by that (its instructions read whole rows)
        if ok:
            ok = not any(_overwrites(o, (op.x, op.weight)) for o in ops[i + 1:users[-1] + 1])
        if not ok:
            continue
        for j in users:
            ops[j] = ops[j].clone(x=op.x, norm_w=op.weight, rms_eps=float(op.eps))
        drop.add(i)
    out.ops = [o for i, o in enumerate(ops) if i not in drop]
    return out


def fuse_rope_attention(g: Graph) -> Graph:
    out = g.derive()
    ops: list[Op] = []
    for i, op in enumerate(g.ops):
        prev = ops[-1] if ops else None
        if (op.kind == "DecodeAttention" and op.k_new is None and prev is not None and prev.kind == "RopeAppend"
                and op.q.same(prev.q_out) and op.k_cache.same(prev.k_cache) and op.v_cache.same(prev.v_cache)
                and op.pos.same(prev.pos) and prev.q_out.buf.kind == "temp" and not _overwrites(op, prev.reads)
                and not _reads_buffer(g.ops[i + 1:], prev.q_out.buf, g.outputs)):
            H, KVH, D = prev.heads, prev.kv_heads, prev.head_dim
            qkv = prev.qkv
            ops[-1] = op.clone(q=qkv.cols_slice(0, H * D), k_new=qkv.cols_slice(H * D, KVH * D),
                               v_new=qkv.cols_slice((H + KVH) * D, KVH * D), cos=prev.cos, sin=prev.sin)
            continue
        ops.append(op)
    out.ops = ops
    return out


def kv_splits(pairs: int, max_seq: int, sm_count: int, head_dim: int = 64) -> int:
    """Instructions per (sequence, kv head) pair: the split count with the lowest modelled time
    waves x (fixed cost per instruction [+ partials and merge when split] + key tiles per split x time per tile),
    with constants measured on B200 (config.DEC_*).  The kernel works in tiles of 128 keys (64 for
    head_dim 128), so splitting below one tile buys nothing and only adds partials to merge.  Few
    pairs (batch 1) spread over one wave of SMs; many pairs stay unsplit until the cache is long
    enough to pay for the partials.  A split keeps at least MIN_SPLIT_KEYS keys of room.
    MEGACUTE_B200_KV_SPLITS overrides the choice (experiments)."""
    cap = max(1, min(max_seq // C.MIN_SPLIT_KEYS, C.MAX_KV_SPLITS))
    if os.environ.get("MEGACUTE_B200_KV_SPLITS"):
        return max(1, min(cap, int(os.environ["MEGACUTE_B200_KV_SPLITS"])))
    tile = 128 if head_dim <= 64 else 64
    best, best_cost = 1, float("inf")
    for s in range(1, cap + 1):
        waves = -(-(pairs * s) // sm_count)
        tiles = -(-(-(-max_seq // s)) // tile)
        merge = C.DEC_MERGE_US + C.DEC_MERGE_US_PER_SPLIT * s if s > 1 else 0.0
        cost = waves * (C.DEC_FIXED_US + merge + tiles * C.DEC_TILE_US)
        if cost < best_cost - 1e-9:
            best, best_cost = s, cost
    return best


def kv_heads_per_instruction(pairs: int, kv_heads: int, max_seq: int, sm_count: int, head_dim: int = 64) -> int:
    """Unsplit decode attention with more (sequence, kv head) pairs than SMs (batched decode): how many
    kv heads of a sequence one instruction handles, one after the other.  An instruction's fetch,
    dependency wait and arrival are paid once, so fewer and longer instructions win as long as they
    still fill the SMs evenly: waves x (shared cost + heads x (per-head cost + tiles x time per tile)).
    MEGACUTE_B200_ATT_HEADS overrides the choice (experiments)."""
    if os.environ.get("MEGACUTE_B200_ATT_HEADS"):
        h = int(os.environ["MEGACUTE_B200_ATT_HEADS"])
        return h if h >= 1 and kv_heads % h == 0 else 1
    tiles = -(-max_seq // (128 if head_dim <= 64 else 64))
    best, best_cost = 1, float("inf")
    for h in (1, 2, 4, 8):
        if kv_heads % h:
            continue
        waves = -(-(pairs // h) // sm_count)
        cost = waves * (C.DEC_SHARED_US + h * (C.DEC_FIXED_US - C.DEC_SHARED_US + tiles * C.DEC_TILE_US))
        if cost < best_cost - 1e-9:
            best, best_cost = h, cost
    return best


def bulk_eligible(op: Op, sm_count: int) -> bool:
    """Can this decode attention run in the many-sequence form (csrc/op_decode_bulk.cuh)?  One warp per
    kv head, head_dim 64, and cache views that are whole rows of their buffers, 128 bytes per kv head,
    so that consecutive rows are one contiguous run of memory.  And should it?  From 32 sequences on, or 8 with long caches; and where the
    per-head form has more instructions (sequence, kv head, split) than SMs, so that they run one behind the other: their fixed cost is there at any
    context, also while the caches are mostly empty.  us a step with full caches and with an eighth of them, per head / whole rows, 8 kv heads: 24
    sequences x 4096 1971 / 1526 and 1326 / 1099, 24 x 2048 1614 / 1283 and 1282 / 1081, 19 x 2048 1534 / 1245 and 1210 / 1073, 13 x 6144 1793 / 1424 and 1310 /
    1095, 10 x 3072 1338 / 1211 and 1130 / 1087, 7 x 8064 1578 / 1362 and 1165 / 1162, unsplit 30 x 4096 2009 / 1747 and 1172 / 1154, 31 x 2048 1544 / 1402 and
    1109 / 1113; 4 kv heads: 20 x 4096 1453 / 1419 and 1170 / 1088.  Unsplit over shorter caches the gain is gone by then (20 x 512 1139 / 1111 and
    1024 / 1058).  A form that fills the SMs once loses by whole rows as soon as caches are not full: 16 x 4096 1451 / 1378, but at a quarter
    1071 / 1149, 8 x 4096 1274 / 1232 and 1049 / 1128, 5 x 12032 1496 / 1389 and 1067 / 1164; 4 kv heads, 31 x 2048 full 1221 / 1372."""
    if os.environ.get("MEGACUTE_B200_ATT_BULK") == "0" or getattr(op, "window", 0):      # (no sliding window in that form)
        return False
    whole = all(v.col0 == 0 and v.cols == v.buf.cols for v in (op.k_cache, op.v_cache))
    ok = op.head_dim == 64 and op.kv_heads <= C.COMPUTE_WARPS and whole and op.k_cache.cols == op.kv_heads * 64
    if os.environ.get("MEGACUTE_B200_ATT_BULK") == "1":
        return ok
    if op.batch >= C.BULK_MIN_BATCH or (op.batch >= C.BULK_MIN_BATCH_LONG and op.max_seq >= C.BULK_LONG_SEQ):
        return ok
    pairs = op.batch * op.kv_heads
    return ok and op.batch >= C.BULK_MIN_BATCH_FEW and op.max_seq >= C.BULK_MIN_SEQ and pairs * kv_splits(pairs, op.max_seq, sm_count) > sm_count


def bulk_kv_splits(batch: int, kv_heads: int, max_seq: int, sm_count: int) -> int:
    """KV splits per sequence in the many-sequence form: the count with the lowest modelled time
    rounds x (cost per instruction + 16-row tiles per split x time per tile), rounds = instructions per
    SM.  Long contexts want enough instructions to fill the last round evenly (batch 64: 2 splits
    leave 20 SMs idle, 9 splits fill 3.9 rounds of 4); the measured cost per instruction grows with
    the split count, which caps it.  MEGACUTE_B200_KV_SPLITS overrides the choice."""
    cap = max(1, min(max_seq // C.MIN_SPLIT_KEYS, C.MAX_KV_SPLITS))
    if os.environ.get("MEGACUTE_B200_KV_SPLITS"):
        return max(1, min(cap, int(os.environ["MEGACUTE_B200_KV_SPLITS"])))
    cost = lambda s: bulk_split_cost(batch, kv_heads, max_seq, sm_count, s)
    return min(range(1, cap + 1), key=lambda s: (round(cost(s), 9), s))


def bulk_split_cost(batch: int, kv_heads: int, max_seq: int, sm_count: int, s: int) -> float:
    """Modelled time (us) of the many-sequence form with s equal splits per sequence."""
    tile_us = C.BULK_TILE_US_PER_KB * kv_heads * 128 / 1024
    tiles = -(-(-(-max_seq // s)) // C.BULK_TILE_ROWS)
    return -(-(batch * s) // sm_count) * (max(C.BULK_FIXED_US, C.BULK_US_PER_SPLIT * s - 3.0) + tiles * tile_us)


def shares_pay(batch: int, splits: int, sm_count: int) -> bool:
    """Instead of `splits` equal splits of each sequence, the same amount of keys on every SM (bulk_kv_shares)?  Where equal splits run in
    several rounds of the SMs: then two instructions per SM cost no more than they did, at any context.  us a step, equal splits / the same
    amount, full caches and an eighth of them: 60 sequences x 4096 rows (7 splits) 2664 / 2315 and 1620 / 1358, 50 x 2048 (5) 1807 / 1624 and 1335 / 1282, 40 x
    4096 (7) 2072 / 1872 and 1377 / 1312, 42 x 2048 (7) 1665 / 1511 and 1335 / 1256, 58 x 2048 (5) 1830 / 1711 and 1353 / 1300, 96 x 4096 (3) 3186 / 3122 and 1558 / 1492, 200 x
    1024 (2) 2862 / 2662 and 2011 / 1878; 4 kv heads: 60 x 4096 (7) 2528 / 2219 and 1597 / 1327.  In one round the second instruction of some SMs is a fixed
    cost that only full caches pay for: 64 x 4224 (2) 2534 / 2462 full, 1831 / 1839 at a half, 1473 / 1532 at a quarter, 1300 / 1389 at an eighth; 44 x 4096 (3)
    2010 / 1959, but 1211 / 1295; 32 x 8192 of 4 heads 2325 / 2303, but 1230 / 1283.  Unsplit sequences in several rounds gain nothing: 296 x 512 2619 / 2614,
    300 x 256 2483 / 2402, at an eighth 2141 / 2165."""
    return splits > 1 and batch * splits > sm_count


@functools.lru_cache(maxsize=256)
def bulk_kv_shares(batch: int, kv_heads: int, max_seq: int, sm_count: int) -> tuple:
    """(modelled time, instructions) of the many-sequence form with the same amount of work on every SM: the sequences' keys, one behind
    the other, are dealt out to the SMs, so that an SM may end one sequence and begin another, with an instruction for each.  Instructions
    are (sequence, split, begin and end in 1024ths of its keys, splits of the sequence), in rounds: an SM's first, its second.

    A second instruction on an SM costs more than a first (BULK_SHARE_US 3 / 5 / 7 / 8: 50 sequences at 2000 -- / 1709 / 1677 / 1639 us a step), so SMs
    with two get fewer keys.  (When: shares_pay.)"""
    whole = -(-max_seq // C.BULK_TILE_ROWS) * C.BULK_TILE_US_PER_KB * kv_heads * 128 / 1024       # us of a sequence
    least = 32                                                                                   # 1024ths
    best = (float("inf"), ())
    low, high = 0.0, 2 * (batch * (whole + C.BULK_SHARE_US) / sm_count + C.BULK_SHARE_US)
    for _ in range(30):                                      # the smallest load of an SM with which they are enough
        budget = (low + high) / 2
        sms, room, load = [[]], budget, [0.0]
        for b in range(batch):
            at = 0
            while at < 1024:
                take = int((room - C.BULK_SHARE_US) / whole * 1024)
                if take < least and sms[-1]:
                    sms.append([])
                    load.append(0.0)
                    room = budget
                    continue
                take = min(max(take, least), 1024 - at)
                if 1024 - at - take < least:
                    take = 1024 - at
                sms[-1].append((b, at, at + take))
                load[-1] += C.BULK_SHARE_US + take / 1024 * whole
                room = budget - load[-1]
                at += take
        if len(sms) <= sm_count:
            high = budget
            if max(load) < best[0]:
                best = (max(load), sms)
        else:
            low = budget
    cost, sms = best
    while 0 < len(sms) < sm_count:                           # (an SM without an instruction would shift the second round)
        at = max(range(len(sms)), key=lambda i: max(u1 - u0 for _, u0, u1 in sms[i]))
        k = max(range(len(sms[at])), key=lambda i: sms[at][i][2] - sms[at][i][1])
        b, u0, u1 = sms[at][k]
        if u1 - u0 < 2 * least:
            return float("inf"), ()
        sms[at][k] = (b, u0, (u0 + u1) // 2)
        sms.append([(b, (u0 + u1) // 2, u1)])
    pieces = sorted(x for sm in sms for x in sm)
    first = {b: k for k, (b, _, _) in reversed(list(enumerate(pieces)))}
    count = {b: sum(x[0] == b for x in pieces) for b in first}
    number = {x: k - first[x[0]] for k, x in enumerate(pieces)}
    sms = sorted(([(x[0], number[x], x[1], x[2], count[x[0]]) for x in sm] for sm in sms), key=len, reverse=True)
    cost += max(0.0, C.BULK_US_PER_SPLIT * max(count.values()) - 3.0 - C.BULK_FIXED_US)
    return cost, tuple(sm[k] for k in range(len(sms[0])) for sm in sms if k < len(sm))


def split_kv(g: Graph, sm_count: int) -> Graph:
    out = g.derive()
    ops = []
    for op in g.ops:
        if op.kind == "DecodeAttention" and op.splits == 1 and bulk_eligible(op, sm_count):
            s = bulk_kv_splits(op.batch, op.kv_heads, op.max_seq, sm_count)
            op = op.clone(heads_per_inst=op.kv_heads, bulk=True)
            if shares_pay(op.batch, s, sm_count) and not os.environ.get("MEGACUTE_B200_KV_SPLITS") and op.max_seq < C.BULK_SHARE_MAX_SEQ:
                shares = bulk_kv_shares(op.batch, op.kv_heads, op.max_seq, sm_count)[1]
                if shares and max(x[4] for x in shares) <= C.MAX_KV_SPLITS:
                    op, s = op.clone(shares=shares), max(x[4] for x in shares)
            if s > 1:
                G, D = op.heads // op.kv_heads, op.head_dim
                cols = -(-(G * D + 2 * G) // 4) * 4          # per (kv head, split): O (G x D), running max (G), sum (G)
                part = out.workspace((op.batch * op.kv_heads * s, cols), torch.float32)
                count = out.workspace((op.batch * op.kv_heads, 1), torch.int32)
                op = op.clone(splits=s, part=part, count=count)
            ops.append(op)
            continue
        if op.kind == "DecodeAttention" and op.splits == 1:
            pairs = op.batch * op.kv_heads
            s = kv_splits(pairs, op.max_seq, sm_count, op.head_dim)
            if s == 1 and (pairs > sm_count or os.environ.get("MEGACUTE_B200_ATT_HEADS")):
                hpi = kv_heads_per_instruction(pairs, op.kv_heads, op.max_seq, sm_count, op.head_dim)
                if hpi > 1:
                    op = op.clone(heads_per_inst=hpi)
            if s > 1:
                G, D = op.heads // op.kv_heads, op.head_dim
                cols = -(-(G * D + 2 * G) // 4) * 4          # per split: O (G x D), running max (G), sum (G)
                s = min(s, C.DECODE_MERGE_BYTES // (cols * 4))   # the merging split holds all partial rows in shared memory
                if s < 2:
                    ops.append(op)
                    continue
                part = out.workspace((pairs * s, cols), torch.float32)
                count = out.workspace((pairs, 1), torch.int32)
                op = op.clone(splits=s, part=part, count=count)
        ops.append(op)
    out.ops = ops
    return out


def _retarget(v, alias):
    if v is None or v.buf.id not in alias:
        return v
    r = alias[v.buf.id]
    return View(r.buf, r.row0 + v.row0, r.col0 + v.col0, v.rows, v.cols)


def choose_k_splits(M: int, N: int, K: int, sm_count: int, finalize: bool) -> int:
    """Split count for a tile GEMM.  Cost of a plan = waves x (fixed cost per instruction + operand
    bytes of one instruction at one SM's share of HBM bandwidth).  Even splits only: six or nine of uneven length, which fill
    144 of 148 SMs where four or eight fill 96 or 128, cost in reduce-adds what they save in streaming (batch-64 decode 0.2 %
    slower).  A SplitFinalize behind the op is a dependency hop of its own (adaLN modulations of 32 images, K = 1024: two splits
    and it 14 us, one instruction per tile 10)."""
    bm, bn, bk = C.GEMM_BM, C.GEMM_BN, C.GEMM_BK
    mt, nt, kt = -(-M // bm), -(-N // bn), K // bk
    rows = min(M, bm)

    def cost(n_inst, k):
        return -(-n_inst // sm_count) * (C.INST_US + (bn + rows) * k * 2 / (C.SM_GBPS * 1e3))

    best, best_cost = 1, cost(mt * nt, K)
    if mt * nt >= sm_count:
        return 1
    for s in range(2, C.MAX_K_SPLITS + 1):
        if kt % s or kt // s < C.MIN_SPLIT_KTILES:
            continue
        c = cost(mt * nt * s, K // s) + (C.FINALIZE_US if finalize else 0.0)
        if c < best_cost:
            best, best_cost = s, c
    return best


def plan_tiles(M: int, N: int, K: int, sm_count: int, max_splits: int, finalize: bool) -> tuple:
    """(K splits, tile rows, tile columns) of a tile linear with more than WIDE_MIN_ROWS rows: the plan with the lowest
    modelled time  rounds x (k-tiles x time per k-tile + time per tile) + time per op [+ reduce-adds, and the
    SplitFinalize behind them], rounds = instructions per SM, with constants from the kernel's timeline
    (config.GEMM_COST_US).  Tiles of 256 rows -- 256 x 256 or 256 x 128 -- are the form whose epilogue runs beside the next
    tile's main loop and whose operands cost fewer bytes per flop (csrc/op_gemm_tc_wide.cuh)."""
    best, best_cost = (1, C.GEMM_BM, C.GEMM_BN), float("inf")
    for (bm, bn), (tile, k, once) in C.GEMM_COST_US.items():
        if bm != C.GEMM_BM and N % bn:
            continue
        for s in range(1, max_splits + 1):
            if (s > 1 and K // s < C.MIN_SPLIT_KTILES * C.GEMM_BK) or (bm != C.GEMM_BM and K % 64):
                continue
            rounds = -(-(-(-M // bm) * -(-N // bn) * s) // sm_count)
            cost = rounds * (-(-(K / 64) // s) * k + tile) + once + (M * N * s * 4 / (C.REDUCE_GBPS * 1e3) + (C.FINALIZE_US if finalize else 0.0) if s > 1 else 0.0)
            if cost < best_cost - 1e-9:
                best, best_cost = (s, bm, bn), cost
    return best


def split_k(g: Graph, sm_count: int) -> Graph:
    out = g.derive()
    alias: dict[int, View] = {}      # id of a dropped output buffer -> residual view that now holds it
    ops: list[Op] = []
    src = list(g.ops)
    for i, op0 in enumerate(src):
        op = op0.clone(**{k: _retarget(v, alias) for k, v in op0.view_fields()}) if alias else op0
        if op.kind == "Linear" and op.act != "swiglu" and not gemv_eligible(op.x.rows, op.x.cols):
            M, K = op.x.shape
            r = op.residual
            whole = op.out.rect == (0, op.out.buf.rows, 0, op.out.buf.cols)
            inplace = (r is not None and op.bias is None and op.act is None and op.norm_w is None
                       and r.buf.kind == "temp" and op.out.buf.kind == "temp" and whole
                       and all(v.buf is not r.buf for v in (op.x, op.w))       # (other instructions still read those)
                       # nobody needs the residual as it was, under its own name or under that of an output added into it before,
                       # and nobody puts anything else there
                       and not any(_retarget(v, alias).buf is r.buf for o in src[i + 1:] for v in o.reads + o.writes))
            if M > C.WIDE_MIN_ROWS:
                s = plan_tiles(M, op.w.rows, K, sm_count, C.MAX_K_SPLITS, not inplace)[0]
            else:
                # (the fused decode attention reads the sums itself: fuse_finalize_attention)
                hop = not inplace and not any(o.kind in ("RopeAppend", "DecodeAttention") and any(v.buf is op.out.buf for v in o.reads) for o in src[i + 1:])
                s = choose_k_splits(M, op.w.rows, K, sm_count, hop)
            if s > 1:
                if inplace:
                    alias[op.out.buf.id] = r
                    new = Op("LinearSplit", x=op.x, w=op.w, ws=r, splits=s)
                    new.layer = op.layer
                    ops.append(new)
                    continue
                ws = out.workspace(op.out.shape, torch.float32)
                part = Op("LinearSplit", x=op.x, w=op.w, ws=ws, splits=s)
                fin = Op("SplitFinalize", ws=ws, out=op.out, bias=op.bias, act=op.act, residual=op.residual)
                part.layer = fin.layer = op.layer
                ops += [part, fin]
                continue
        ops.append(op)
    out.ops = ops
    out.outputs = [_retarget(v, alias) for v in g.outputs]
    return out


def _accepts(op: Op, field: str, dtype) -> bool:
    """Can the kernel read / write operand `field` of `op` in `dtype` (fp32 or fp16) instead of bf16?"""
    k = op.kind
    f32 = dtype == torch.float32
    if k == "Linear":
        streaming = gemv_eligible(op.x.rows, op.x.cols)
        if field == "x":                                # the tensor core takes 16-bit operands; the streaming linear converts
            return streaming or not f32
        return field in ("out", "residual") or (field == "gate" and (op.bm == C.GEMM_BM_WIDE or not f32))
    if k == "LinearSplit":
        return (field == "ws" and f32) or (field == "x" and not f32)
    if k == "SplitFinalize":
        return field in ("out", "residual", "gate") or (field == "ws" and f32)
    if k == "Norm":
        return field in ("x", "out")
    if k in ("Unary", "Binary", "SwiGLU", "Modulate"):
        return True
    if k == "Rope":
        return field in ("x", "out")
    if k == "Attention":                              # (q, k and v must end up with one dtype: promote_temps checks the trio)
        return not f32
    if k == "RopeAppend":
        return field == "qkv"
    if k == "Gather":
        return field == "out"
    if k == "Argmax":
        return field == "x"
    if k == "DecodeAttention":
        if field in ("q", "k_new", "v_new"):          # one dtype code covers all three
            return op.k_new is None or (op.q.buf is op.k_new.buf is op.v_new.buf)
        return field == "out"
    return False


# runtime-private activations up to this size are kept in fp32 when every op touching them can; larger
# ones (prefill, DiT: megabytes per tensor, streamed through L2 by bandwidth-bound pointwise ops) in fp16
F32_TEMP_BYTES = 4 << 20


def promote_temps(g: Graph) -> Graph:
    """Keep runtime-private activations in more than bf16's 8 significant bits wherever every op that
    touches them can: the residual stream, the QKV row, the attention output and the MLP hidden of a
    step are never seen by the caller, and rounding each of them to bf16 at every layer is the main
    source of drift against an fp32 evaluation (16 layers of the 1B shape: 1.5e-2 to 2.5e-2 rel-L2 on
    the logits with bf16 intermediates, ~2e-3 without).  fp32 for small tensors when every user
    accepts it (decode); otherwise fp16 -- the same bytes as bf16, 11 significant bits, accepted by the
    tensor cores as the A operand of a tile GEMM beside bf16 weights; conversions saturate at +-65504.
    Buffers the caller sees (inputs, params, states, outputs) keep their dtype.
    MEGACUTE_B200_BF16_TEMPS=1 leaves every temp in bf16."""
    out = g.derive()
    if os.environ.get("MEGACUTE_B200_BF16_TEMPS") == "1":
        return out
    users: dict[int, list] = {}
    for op in g.ops:
        for name, v in op.view_fields():
            users.setdefault(v.buf.id, []).append((op, name))
    # the residual stream that K splits reduce-add into, however large: added in bf16, eight partial sums per layer are rounded to
    # eight bits one by one (measured: 4 layers of the 1B shape over 600 tokens, logits 1.5e-2 rel-L2 apart from one run to the next)
    accumulated = {op.ws.buf.id for op in g.ops if op.kind == "LinearSplit"}
    swap: dict[int, Buffer] = {}
    for b in g.buffers:
        if b.kind != "temp" or b.dtype != torch.bfloat16 or b.id not in users:
            continue
        if any(v.buf is b for v in g.outputs):
            continue
        for dt in (torch.float32, torch.float16):
            if dt == torch.float32 and b.rows * b.cols * 4 > F32_TEMP_BYTES and b.id not in accumulated:
                continue
            if all(_accepts(op, name, dt) for op, name in users[b.id]):
                swap[b.id] = Buffer(b.name, b.rows, b.cols, dt, "temp")
                break
    # an attention's q, k and v share one dtype (one tensor-core instruction takes one operand type): a trio of
    # which not every member changes to fp16 stays as it was
    changed = True
    while changed:
        changed = False
        for op in g.ops:
            if op.kind != "Attention":
                continue
            new = [swap[v.buf.id].dtype if v.buf.id in swap else v.buf.dtype for v in (op.q, op.k, op.v)]
            if len(set(new)) > 1:
                for v in (op.q, op.k, op.v):
                    if swap.pop(v.buf.id, None) is not None:
                        changed = True
    if not swap:
        return out
    move = lambda v: View(swap[v.buf.id], v.row0, v.col0, v.rows, v.cols) if v is not None and v.buf.id in swap else v
    out.ops = [op.clone(**{k: move(v) for k, v in op.view_fields()}) for op in g.ops]
    out.buffers = [swap.get(b.id, b) for b in g.buffers]
    return out


def fuse_finalize_attention(g: Graph) -> Graph:
    """A split-K QKV projection leaves its sums in an fp32 workspace; when the SplitFinalize behind it
    is a plain copy (no bias, activation or residual, fp32 output) whose only reader is the fused
    decode attention, the attention reads the workspace itself and zeroes what it has read (the
    finalize's other duty), and the copy -- a dependency hop of ~9 us per layer in batched decode --
    is dropped."""
    if os.environ.get("MEGACUTE_B200_KEEP_FINALIZE"):
        return g
    out = g.derive()
    ops: list[Op] = []
    for i, op in enumerate(g.ops):
        prev = ops[-1] if ops else None
        if (op.kind == "DecodeAttention" and op.k_new is not None and prev is not None and prev.kind == "SplitFinalize"
                and prev.bias is None and prev.act is None and prev.residual is None
                and prev.out.buf.kind == "temp" and prev.out.buf.dtype == torch.float32
                and all(v.buf is prev.out.buf and v.rows == prev.out.rows and prev.out.row0 == v.row0
                        and prev.out.col0 <= v.col0 and v.col0 + v.cols <= prev.out.col0 + prev.out.cols
                        for v in (op.q, op.k_new, op.v_new))
                and not _reads_buffer(g.ops[i + 1:], prev.out.buf, g.outputs)):
            move = lambda v: prev.ws.cols_slice(v.col0 - prev.out.col0, v.cols)
            ops[-1] = op.clone(q=move(op.q), k_new=move(op.k_new), v_new=move(op.v_new), zero_inputs=True)
            continue
        ops.append(op)
    out.ops = ops
    return out


def wide_tiles(g: Graph, sm_count: int) -> Graph:
    """Output tile of every tile linear with more than WIDE_MIN_ROWS rows (plan_tiles, with the K splits split_k chose).
    MEGACUTE_B200_WIDE_TILES=0 / 1 forces 128 x 128 / 256 x 256 where the shape allows it."""
    force = os.environ.get("MEGACUTE_B200_WIDE_TILES")
    out = g.derive()
    ops = []
    for op in g.ops:
        if op.kind in ("Linear", "LinearSplit") and not gemv_eligible(op.x.rows, op.x.cols) and not op.bn:
            M, K = op.x.shape
            N = op.w.rows
            splits = op.splits if op.kind == "LinearSplit" else 1
            if M > C.WIDE_MIN_ROWS and K % 64 == 0 and force != "0":
                # (a split op is planned as `splits` independent products over K / splits)
                _, bm, bn = plan_tiles(M, N, -(-K // 64 // splits) * 64, max(1, sm_count // splits), 1, False)
                if force == "1" and N % C.GEMM_BN_WIDE == 0:
                    bm, bn = C.GEMM_BM_WIDE, C.GEMM_BN_WIDE
                if bm != C.GEMM_BM:
                    op = op.clone(bm=bm, bn=bn)
        ops.append(op)
    out.ops = ops
    return out


def halve_last_tiles(g: Graph, sm_count: int) -> Graph:
    """A linear of 256 x 256 tiles that occupies at most three quarters of the SMs with one tile each: its last row blocks become a linear
    of their own with 256 x 128 tiles, as many blocks as the free SMs hold.  The first row blocks' operands are there before the op in front
    has ended, so the SMs that are free by then take a whole tile and the others, which come later, half of one (two thirds of its time).
    3001 rows, N = 2048, K = 5632: all 96 tiles end after 68 us on 96 SMs, the 32 that start last 25 us behind the rest; now 54 us on 144.
    MLP block of 2400 / 2700 / 3001 rows 164 -> 158, 184 -> 173, 188 -> 181 us, 4 layers of 2900 tokens (K = 8192) 1923 -> 1883.
    That needs a linear of at least as many products in front: with x from outside the launch all tiles start together (alone, 2500 rows, K = 8192 97.1 ->
    99.8), and behind a short one nearly so (K = 512 in front, 3000 rows, K = 5632 107.6 -> 109.3).
    With more tiles (128: MLP of 4096 rows 230 both ways) too few SMs are free.  Half tiles move a third more operand bytes per flop, so
    that short products lose where the op behind fills the gap anyway: K = 4096 (DiT of 24 images) 6443 -> 6472, any K 6438 -> 6517."""
    out = g.derive()
    ops = []
    for op in g.ops:
        r = 0
        if op.kind == "Linear" and (op.bm, op.bn) == (C.GEMM_BM_WIDE, C.GEMM_BN_WIDE) and op.cos is None and op.x.cols > C.HALVE_MIN_COLS:
            M, group = op.x.rows, 1 if op.gate is None else op.gate_group
            mt, nt = -(-M // op.bm), op.w.rows // op.bn
            front = next((o for o in reversed(ops) if any(v.buf is op.x.buf for v in o.writes)), None)
            behind = front is not None and front.kind == "Linear" and front.w.rows * front.w.cols >= op.w.rows * op.w.cols
            r = min(mt - 1, (sm_count - mt * nt) // nt) if behind and 4 * mt * nt <= 3 * sm_count else 0
            m0 = (mt - r) * op.bm
        if r <= 0 or m0 % group or M - m0 <= C.WIDE_MIN_ROWS or os.environ.get("MEGACUTE_B200_WIDE_TILES"):
            ops.append(op)
            continue
        for a, rows, bn in ((0, m0, op.bn), (m0, M - m0, C.GEMM_BN)):
            cut = {f: getattr(op, f).rows_slice(a, rows) for f in ("x", "out", "residual") if getattr(op, f) is not None}
            if op.gate is not None:
                cut["gate"] = op.gate.rows_slice(a // group, rows // group)
            ops.append(op.clone(bn=bn, **cut))
    out.ops = ops
    return out


def split_argmax(g: Graph, sm_count: int) -> Graph:
    """An argmax over few long rows is cut into column chunks, about two instructions per SM in all;
    every chunk leaves its best (value, index) in a workspace and the last chunk of a row to arrive
    picks the winner (the scheme of the split decode attention)."""
    out = g.derive()
    ops = []
    for op in g.ops:
        if op.kind == "Argmax" and op.part is None:
            rows, cols = op.x.shape
            chunks = max(1, min(C.ARGMAX_MAX_CHUNKS, -(-2 * sm_count // rows), cols // 1024))
            if chunks > 1:
                # per row: the chunks' best values, then (from a 16-byte boundary on) the bits of their indices
                op = op.clone(chunks=chunks, part=out.workspace((rows, 2 * (-(-chunks // 4) * 4)), torch.float32),
                              count=out.workspace((rows, 1), torch.int32))
        ops.append(op)
    out.ops = ops
    return out


def fuse_pointwise(g: Graph) -> Graph:
    """Two pointwise pairs of an adaLN block become one op each (no counterpart among the reference's passes; its graphs
    run them as written, examples/dit/model.py):

    * ``Norm -> Modulate``: ``norm(x) * (1 + scale[g]) + shift[g]`` in the norm's own pass over the row;
    * ``Binary(mul, y, gate[g]) -> Binary(add, x, .)``: ``x + y * gate[g]`` (a gated residual).

    Each pair's intermediate is a runtime-private tensor nothing else reads.  A pointwise op over an activation costs
    one read and one write of it plus a dependency hop: a DiT block drops from eight such ops to four.
    MEGACUTE_B200_NO_POINTWISE_FUSION=1 keeps the ops apart."""
    if os.environ.get("MEGACUTE_B200_NO_POINTWISE_FUSION") == "1":
        return g
    out = g.derive()
    ops: list[Op] = []
    for i, op in enumerate(g.ops):
        prev = ops[-1] if ops else None
        private = lambda v: v.buf.kind == "temp" and not _reads_buffer(g.ops[i + 1:], v.buf, g.outputs)
        if (op.kind == "Modulate" and prev is not None and prev.kind == "Norm" and prev.scale is None
                and op.x.same(prev.out) and private(prev.out) and all(v.buf is not prev.out.buf for v in (op.scale, op.shift))
                and not _overwrites(op, (prev.weight, prev.bias), in_place=prev.x)):
            ops[-1] = prev.clone(out=op.out, scale=op.scale, shift=op.shift, group=op.group)
            continue
        if (op.kind == "Binary" and op.fn == "add" and op.b_group == 1 and op.gate is None and prev is not None
                and prev.kind == "Binary" and prev.fn == "mul" and prev.gate is None and prev.b_group > 1
                and not _overwrites(op, (prev.b,), in_place=prev.a)):
            for mine, other in ((op.b, op.a), (op.a, op.b)):
                if mine.same(prev.out) and private(prev.out) and other.shape == op.out.shape and other.buf is not prev.out.buf:
                    ops[-1] = op.clone(a=other, b=prev.a, gate=prev.b, gate_group=prev.b_group)
                    break
            else:
                ops.append(op)
            continue
        ops.append(op)
    out.ops = ops
    return out


def fuse_gated_linear(g: Graph) -> Graph:
    """A tile linear -- or the SplitFinalize behind its K splits -- followed by a gated residual (``x + y * gate[g]``, made by fuse_pointwise) does the gating in its epilogue: a
    pass over three activation-sized tensors and a dependency hop less (7 us per hop in a DiT block of 1024 rows), and the
    product is not rounded in between.  (128-row tiles take a 16-bit gate only; streaming linears keep the op.)
    MEGACUTE_B200_NO_POINTWISE_FUSION=1 keeps the ops apart."""
    if os.environ.get("MEGACUTE_B200_NO_POINTWISE_FUSION") == "1":
        return g
    out = g.derive()
    ops: list[Op] = []
    for i, op in enumerate(g.ops):
        prev = ops[-1] if ops else None
        if (op.kind == "Binary" and op.gate is not None and op.fn == "add" and prev is not None
                and (prev.kind == "SplitFinalize" or (prev.kind == "Linear" and (
                    prev.bm == C.GEMM_BM_WIDE or (not gemv_eligible(prev.x.rows, prev.x.cols) and op.gate.buf.dtype != torch.float32))))
                and prev.act != "swiglu" and prev.residual is None and prev.gate is None
                and op.b.same(prev.out) and prev.out.buf.kind == "temp" and not _reads_buffer(g.ops[i + 1:], prev.out.buf, g.outputs)
                # (the product is not stored any more: neither the residual nor the gate may be it)
                and op.a.buf is not prev.out.buf and op.gate.buf is not prev.out.buf
                and not _overwrites(op, prev.reads)):
            ops[-1] = prev.clone(out=op.out, residual=op.a, gate=op.gate, gate_group=op.gate_group)
            continue
        ops.append(op)
    out.ops = ops
    return out


def fuse_rope_linear(g: Graph) -> Graph:
    """A tile linear whose leading output columns are read only by Ropes whose results go to prefill attention rotates them in
    its epilogue: the heads lie whole in a tile and the fp32 accumulators are at hand, so two passes over q and k, their
    dependency hop and a rounding go.  q and k stay where they are, side by side with v.  (With head_dim 64 or 128, 16-bit tables and
    nothing else between product and rotation: what the epilogues know.)  MEGACUTE_B200_NO_POINTWISE_FUSION=1 keeps the ops apart."""
    if os.environ.get("MEGACUTE_B200_NO_POINTWISE_FUSION") == "1":
        return g
    out = g.derive()
    ops = list(g.ops)
    alias: dict[int, View] = {}
    fused: dict[int, Op] = {}
    for i, lin in enumerate(ops):
        if (lin.kind != "Linear" or gemv_eligible(lin.x.rows, lin.x.cols) or lin.act is not None or lin.bias is not None
                or lin.residual is not None or lin.gate is not None or lin.rms_eps is not None):
            continue
        buf = lin.out.buf
        if buf.kind != "temp" or lin.out.rect != (0, buf.rows, 0, buf.cols) or any(v.buf is buf for v in g.outputs):
            continue
        ropes = [k for k in range(i + 1, len(ops)) if ops[k].kind == "Rope" and ops[k].x.buf is buf]
        if not ropes:
            continue
        first, col = ops[ropes[0]], 0
        ok = first.head_dim in (64, 128) and first.cos.buf.dtype != torch.float32
        for k in sorted(ropes, key=lambda k: ops[k].x.col0):
            r = ops[k]
            ok = (ok and r.x.rect == (0, buf.rows, col, col + r.x.cols) and r.x.cols == r.heads * r.head_dim
                  and r.cos.same(first.cos) and r.sin.same(first.sin) and (r.seq, r.head_dim) == (first.seq, first.head_dim)
                  and r.cos.buf.dtype == r.sin.buf.dtype and r.out.buf.kind == "temp" and r.out.buf is not buf
                  and r.out.rect == (0, r.out.buf.rows, 0, r.out.buf.cols) and not any(v.buf is r.out.buf for v in g.outputs)
                  and r.out.buf.dtype == buf.dtype       # (attention reads the linear's buffer in its place: fp32 it does not take)
                  and all(o.kind == "Attention" for o in ops if any(v.buf is r.out.buf for v in o.reads))
                  and sum(any(v.buf is r.out.buf for v in o.writes) for o in ops) == 1)
            col += r.x.cols
        # nothing else touches the columns that are now rotated in place, and the tables are what they are when the linear runs
        for k, o in enumerate(ops):
            if k != i and k not in ropes:
                ok = ok and not any(v.buf is buf for v in o.writes) and not any(v.buf is buf and v.col0 < col for v in o.reads)
            if i < k < ropes[-1]:
                ok = ok and not any(v.buf is t.buf for v in o.writes for t in (first.cos, first.sin))
        if not ok:
            continue
        fused[i] = lin.clone(cos=first.cos, sin=first.sin, rope_cols=col, head_dim=first.head_dim, seq=first.seq)
        for k in ropes:
            alias[ops[k].out.buf.id] = ops[k].x
            fused[k] = None
    out.ops = []
    for i, op in enumerate(ops):
        op = fused.get(i, op)
        if op is not None:
            out.ops.append(op.clone(**{k: _retarget(v, alias) for k, v in op.view_fields()}) if alias else op)
    return out


def direct_buffers(g: Graph) -> frozenset:
    """Ids of the runtime-private fp32 buffers that need no dependency counters because their readers look at the values
    themselves (csrc/mk_device.cuh: direct operands): written whole by one op that can mark its stores -- a streaming linear, the
    per-head decode attention, an embedding gather -- and read only by ops that can wait for values: streaming linears (x,
    residual) and the per-head decode attention (q, k_new, v_new).  In a step of few rows that is every hop but those through
    a K-split linear."""
    from .encode import gemv_units
    streaming = lambda op: op.kind == "Linear" and gemv_eligible(op.x.rows, op.x.cols) and gemv_units(op)
    per_head = lambda op: op.kind == "DecodeAttention" and not op.bulk and not op.zero_inputs
    users: dict[int, list] = {}
    for k, op in enumerate(g.ops):
        for name, v in op.view_fields():
            users.setdefault(v.buf.id, []).append((k, op, name, v))
    outs = {v.buf.id for v in g.outputs}
    direct = set()
    for b in g.buffers:
        if b.kind != "temp" or b.dtype != torch.float32 or b.id in outs or b.id not in users:
            continue
        writers = [u for u in users[b.id] if any(v.buf is b for v in u[1].writes) and u[2] in ("out", "ws")]
        readers = [u for u in users[b.id] if u not in writers]
        if len(writers) != 1 or not readers or any(v.buf is b for v in writers[0][1].reads):
            continue
        k, op, name, v = writers[0]
        ok = name == "out" and v.rect == (0, b.rows, 0, b.cols) and (streaming(op) or per_head(op) or op.kind == "Gather")
        for j, r, field, _ in readers:
            ok = ok and j > k and not any(w.buf is b for w in r.writes) and (
                (streaming(r) and field in ("x", "residual"))
                or (per_head(r) and r.k_new is not None and field in ("q", "k_new", "v_new") and r.q.buf is r.k_new.buf is r.v_new.buf))
        if ok:
            direct.add(b)
    # (The first linear of a launch has no direct input, so a program with direct hops runs two forms of the streaming linear, and fetches the
    # code of the second one cold, 1 us per launch.  A hop by value gains 0.3 us between narrow linears, 1.5 to 2.5 between wide ones: one or
    # two narrow hops do not pay.  By value / through counters, us per call back to back: one hop of 256 columns 14.5 / 13.4, of 2048 15.1 / 14.6,
    # of 4096 23.5 / 24.8, of 8192 59.3 / 61.6, an MLP block of one row with 5632 25.2 / 26.9; two of 256 17.0 / 16.7, of 2048 19.0 / 18.75, of 4096
    # 31.5 / 33.4; four of 256 24.9 / 24.9, of 2048 28.1 / 29.0.)
    if len(direct) <= 2 and all(b.cols < C.DIRECT_MIN_COLS for b in direct):
        return frozenset()
    return frozenset(b.id for b in direct)


HOIST_MIN_OPS = 4


def hoist_linears(g: Graph) -> Graph:
    """A linear whose operands are ready HOIST_MIN_OPS or more ops before its place moves up behind the last op it depends on.
    An SM runs its instructions in order: the adaLN modulation of a DiT block, which only needs the conditioning vector, cost every
    block its 10 us among ops that wait for one another (its weights cold, half the SMs without a tile); one behind the
    other, the modulations of all blocks stream at the rate of HBM."""
    out = g.derive()
    ops: list[Op] = []
    for op in g.ops:
        j = len(ops)
        if op.kind in ("Linear", "LinearSplit", "SplitFinalize"):
            reads, writes = {v.buf.id for v in op.reads}, {v.buf.id for v in op.writes}
            while j > 0:
                o = ops[j - 1]
                w = {v.buf.id for v in o.writes}
                if w & (reads | writes) or writes & {v.buf.id for v in o.reads}:
                    break
                j -= 1
            if len(ops) - j < HOIST_MIN_OPS:
                j = len(ops)
        ops.insert(j, op)
    out.ops = ops
    return out


def run_all(g: Graph, sm_count: int) -> Graph:
    """The pass pipeline of ``compile`` (reference order: runtime.py:235, plus wide_tiles, split_argmax,
    fuse_pointwise, fuse_gated_linear, fuse_rope_linear, promote_temps, fuse_finalize_attention, hoist_linears and halve_last_tiles)."""
    g = split_argmax(split_kv(fuse_rope_attention(wide_tiles(split_k(fold_norms(g), sm_count), sm_count)), sm_count), sm_count)
    g = hoist_linears(fuse_finalize_attention(promote_temps(fuse_rope_linear(fuse_gated_linear(fuse_pointwise(g))))))
    return halve_last_tiles(g, sm_count)
