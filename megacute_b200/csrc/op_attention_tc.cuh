// MK_OP_ATTENTION on the 5th-generation tensor cores (tcgen05 + tensor memory), head_dim 64 or 128.
// One instruction = (batch b, head h, 256 queries): two tiles of 128 queries that share every K and V tile.  The host
// library selects this body by attaching three tensor maps (q, k, v: {columns, rows}, boxes of 64 columns x 128 rows,
// 128-byte swizzle, zero fill) through ptr 11.
//
//   S = Q_t K_j^T    tcgen05.mma 128 x 128 x 16: Q tile and 128-key tile as K-major operands in shared memory; S in tensor memory
//   softmax          compute warps 4 t .. 4 t + 3, one thread per query row of tile t (a tensor-memory lane): the row's 128 scores are
//                    read twice, 32 at a time, for the maximum and for the exponentials, so nothing is exchanged between
//                    threads.  Log2 domain, scale * log2(e) folded into the subtraction.  The running maximum is only raised
//                    when it grows by more than 2^8 (the reference's lazy rescale, megacute/ops/attention.py:37,252-262): then
//                    the row's sum and its O row in tensor memory are scaled down.
//   O += P V_j       P, rounded to the operand type, goes back to tensor memory, over the scores, as the A operand; V_j as loaded ([key][64 dims])
//                    is the MN-major B operand; O in tensor memory
//   out = O / l      read back, a row per thread; a fully masked row yields 0
// Bound by the special function units: the exponentials of a block of both tiles take 2048 cycles, its products 1024 (head_dim 64)
// or 2048 (128).  What keeps the distance is latency between the roles, so the scores of a block are multiplied ahead: the blocks
// of both tiles are numbered in one sequence, and the scores of block n + 3 (head_dim 128: n + 2) are issued right behind
// block n's P V, into the same tensor-memory buffer, where P lies over the scores.  Products execute in the order of issue, so
// nothing has to be waited for in between, and the tiles fall out of step by themselves: one exponentiates while the other waits.
// Per block of both tiles, 4 x 4096 causal, 32 heads: one buffer a tile, scores requested after P V 5900 cycles; scores first,
// fp32 operations in pairs 4400; three buffers 3600.  (Taken back, each slower: the tiles made to exponentiate in turns with a
// barrier; two 32-column loads in flight.)
//
// Three roles run ahead of one another across the instructions of a run, as in the tile GEMM (op_gemm_tc_wide.cuh):
//   feeder warp      waits for the instruction's dependencies itself, requests Q, then K and V through two stages each
//   issuer warp      the products of both tiles in one fixed order; told by the feeder through Ctrl::wide_info
//   compute warps    softmax and output
// Barriers are initialised once per launch; every role counts.  Tensor memory (columns): three (two) buffers of scores from 0, O of
// both tiles behind them.
// Shared memory: head_dim 64: two Q tiles, two K and two V stages in the work area; head_dim 128: Q in the work area, K and V in the
// ring's memory, which the producer warp grants for a run (Ctrl::ring_granted / ring_returned).
// Every wait is bounded.  Operands the tensor maps cannot describe run the mma.sync body.
//
// ptr 0 q, 1 k, 2 v, 3 out, 11 tensor maps; i 0 batch, 1 seq_q, 2 seq_k, 3 heads, 4 kv_heads, 5 head_dim,
// 6 causal, 7 out dtype, 8 dtype of q, k, v; f 0 scale.  args: 0 b, 1 h, 2 query tile pair.
#pragma once
#include "mk_device.cuh"
#include "tc.cuh"

namespace mk {

constexpr float kAtRescale = 8.0f;                            // raise the running maximum only past 2^8
// byte offsets from the ring's start
template <int D> struct AtMap {
    static constexpr int kTile = 128 * D * 2;                 // one tile of Q, K or V: D / 64 sub-tiles of 128 x 64
    static constexpr int kQ = kRingBytes + kTcXOff;
    static constexpr int kK = D == 64 ? kQ + 2 * kTile : 0;
    static constexpr int kV = kK + 2 * kTile;
    static constexpr uint32_t kScores = D == 64 ? 3 : 2;      // tensor-memory buffers of scores, 128 columns each from column 0
    static constexpr uint32_t kO = kScores * 128;             // ... then O of tile 0 and of tile 1
};
static_assert(AtMap<64>::kV + 2 * AtMap<64>::kTile <= kRingBytes + kWorkBytes, "attention tiles, head_dim 64");
static_assert(AtMap<128>::kV + 2 * AtMap<128>::kTile <= kRingBytes && AtMap<128>::kQ + 2 * AtMap<128>::kTile <= kRingBytes + kWorkBytes, "attention tiles, head_dim 128");

__device__ __forceinline__ int at_blocks(const mk_op_desc* op, int qi, int t) {        // 128-key blocks of tile t (0: no such queries)
    const int q0 = qi * 256 + t * 128;
    if (q0 >= op->i[1]) return 0;
    const int kend = op->i[6] ? min(op->i[2], q0 + 128) : op->i[2];
    return (kend + 127) / 128;
}

// 3-D tiled bulk tensor copy global -> shared without a cache hint: columns, rows of a sequence, sequence.  Rows behind a sequence's last one are zeros
// and not the next sequence's: masked keys have no weight, but what they are multiplied with must be a number (nor need the next
// sequence's rows have been written yet).
__device__ __forceinline__ void tma_load_3d_plain(void* dst, const void* tmap, int x, int y, int z, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                     smem_u32(dst)),
                 "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}
// 32 consecutive fp32 columns of this thread's lane, tensor memory <- registers
__device__ __forceinline__ void tc_st32(uint32_t taddr, const float* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(taddr),
        "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
        "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
        "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
        "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
        "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
        : "memory");
}
// 16 words of this thread's lane (32 values of a 16-bit operand), not waited for
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* w) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]),
        "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D = A B (+ D) with A in tensor memory
__device__ __forceinline__ void tc_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// two fp32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{ .reg .b64 x, y, z, w; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mov.b64 z, {%6, %7}; fma.rn.f32x2 w, x, y, z; mov.b64 {%0, %1}, w; }"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{ .reg .b64 x, y, w; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 w, x, y; mov.b64 {%0, %1}, w; }"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// two fp16 from fp32 of at most 2^8: nothing to saturate
__device__ __forceinline__ uint32_t pack2h_fast(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The blocks of an instruction in the order in which the issuer takes them: the tiles in turns, then what one of them has more.
__device__ __forceinline__ int at_order(int t, int j, int both) { return j < both ? 2 * j + t : both + j; }

// ---- feeder warp ---------------------------------------------------------------------------------------------------------------
struct AtFeed {
    uint32_t go = 0, granted = 0;        // parities of attn_go, ring_granted
    uint32_t insts = 0, tiles = 0;       // instructions and K (V) tiles requested
    uint32_t q = 0, k = 0, v = 0;        // (lane 0) phases armed
};
// Lane 0: parities of the phases last armed, as in armed_parities: q, k (2 bits), v (2 bits).
__device__ __forceinline__ uint32_t at_feed_left(const AtFeed& f) {
    return ((f.q & 1u) ^ 1u) | armed_parities(2, f.k & 1u, (f.k >> 1) & 1u) << 1 | armed_parities(2, f.v & 1u, (f.v >> 1) & 1u) << 3;
}
// Abort path: tiles requested and not yet landed
__device__ __forceinline__ void at_wait_landed(AttnBars* a, uint32_t left) {
    wait_landed(&a->q_full, 1, left);
    wait_landed(a->k_full, 2, left >> 1);
    wait_landed(a->v_full, 2, left >> 3);
}
// All lanes; lane 0 requests.  `first`: the CTA's previous instruction is not an attention of the same head_dim.  `told`: entry of
// Ctrl::wide_info to use (shared with the tile GEMM).
template <int D>
__device__ __forceinline__ bool at_feed(const Params& p, Ctrl* c, uint8_t* ring, const mk_op_desc* op, const Inst& in, bool first, AtFeed& f,
                                        uint32_t told) {
    using M = AtMap<D>;
    const int lane = threadIdx.x & 31;
    const int Sq = op->i[1], hk = in.a1 / (op->i[3] / op->i[4]);
    const int nb0 = at_blocks(op, in.a2, 0), nb1 = at_blocks(op, in.a2, 1), nb = max(nb0, nb1);
    const uint8_t* tmaps = reinterpret_cast<const uint8_t*>(op->ptr[11]);
    AttnBars* a = &c->attn;
    bool ok = true;
    if (first) {
        // the compute warps may be busy with earlier instructions for a long time: twice the time limit, so that a stuck wait there reports first
        if (lane == 0) ok = wait_barrier(p, c, &c->attn_go, f.go, in.seq, WHERE_DEP, 2);
        f.go ^= 1u;
        if (D == 128) {
            if (lane == 0 && ok) ok = wait_barrier(p, c, &c->ring_granted, f.granted, in.seq, WHERE_RING_EMPTY, 2);
            f.granted ^= 1u;
        }
        if (!__all_sync(0xffffffffu, ok)) return false;
    }
    for (int k = lane; k < in.nwait; k += 32) {
        const int2 w = __ldg(p.waits + in.wait_off + k);
        ok = wait_counter(p, c, w.x, w.y, in.seq) && ok;
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    if (lane == 0) {
        // the tiles' memory was last written through the generic proxy, and so were q, k and v, by other SMs
        asm volatile("fence.proxy.async;" ::: "memory");
        ok = wait_barrier(p, c, &a->q_free, (f.insts & 1u) ^ 1u, in.seq, WHERE_RING_EMPTY, 2) &&
             check_phase(p, c, &a->q_full, f.insts & 1u, in.seq, WHERE_CHECK_ARM);
        if (ok) {
            const int qtiles = in.a2 * 256 + 128 < Sq ? 2 : 1;
            mbar_arrive_expect_tx(&a->q_full, (uint32_t)(qtiles * M::kTile));
            ++f.q;
            for (int t = 0; t < qtiles; ++t)
                for (int s = 0; s < D / 64; ++s)
                    tma_load_3d_plain(ring + M::kQ + t * M::kTile + s * kTcTileBytes, tmaps, in.a1 * D + s * 64, in.a2 * 256 + t * 128, in.a0, &a->q_full);
            c->wide_info[told & 3u] = make_int4(-(nb0 | nb1 << 15), D, op->i[8] == DT_F16 ? 1 : 0, in.seq);
            mbar_arrive(&c->wide_told[told & 3u]);
        }
        for (int j = 0; j < nb && ok; ++j) {
            const uint32_t n = f.tiles + (uint32_t)j, u = n & 1u, ph = (n >> 1) & 1u;
            ok = wait_barrier(p, c, &a->k_empty[u], ph ^ 1u, in.seq, WHERE_RING_EMPTY, 2) && check_phase(p, c, &a->k_full[u], ph, in.seq, WHERE_CHECK_ARM);
            if (!ok) break;
            mbar_arrive_expect_tx(&a->k_full[u], (uint32_t)M::kTile);
            ++f.k;
            for (int s = 0; s < D / 64; ++s)
                tma_load_3d_plain(ring + M::kK + u * M::kTile + s * kTcTileBytes, tmaps + 128, hk * D + s * 64, j * 128, in.a0, &a->k_full[u]);
            ok = wait_barrier(p, c, &a->v_empty[u], ph ^ 1u, in.seq, WHERE_RING_EMPTY, 2) && check_phase(p, c, &a->v_full[u], ph, in.seq, WHERE_CHECK_ARM);
            if (!ok) break;
            mbar_arrive_expect_tx(&a->v_full[u], (uint32_t)M::kTile);
            ++f.v;
            for (int s = 0; s < D / 64; ++s)
                tma_load_3d_plain(ring + M::kV + u * M::kTile + s * kTcTileBytes, tmaps + 256, hk * D + s * 64, j * 128, in.a0, &a->v_full[u]);
        }
    }
    ++f.insts;
    f.tiles += (uint32_t)nb;
    return __all_sync(0xffffffffu, ok) != 0;
}

// ---- issuer warp ---------------------------------------------------------------------------------------------------------------
struct AtIssue {
    uint32_t insts = 0, tiles = 0;       // instructions, K / V tiles
    uint32_t blocks[2] = {0, 0};         // blocks of each tile (parities of p_full, pv_done; together: place of the next scores)
    uint32_t outs[2] = {0, 0};           // instructions that had the tile (parity of o_free)
};
// Every lane asks the barrier (the answers can differ while a phase completes: the vote makes the warp take one path).
__device__ __forceinline__ bool at_ready(unsigned long long* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) != 0; }
// The whole warp waits, one elected lane issues.  Returns false when aborting.
template <int D>
__device__ __forceinline__ bool at_issue(const Params& p, Ctrl* c, uint8_t* ring, const int4& info, AtIssue& f) {
    using M = AtMap<D>;
    AttnBars* a = &c->attn;
    const int nbt[2] = {(-info.x) & 0x7fff, (-info.x) >> 15};
    const int both = min(nbt[0], nbt[1]), total = nbt[0] + nbt[1], tail = nbt[1] > nbt[0] ? 1 : 0;
    const uint32_t tmem = *(volatile uint32_t*)&c->tmem_base, first = f.blocks[0] + f.blocks[1];
    const uint32_t fmt = info.z ? 0u : 1u;                    // operand format: 0 fp16, 1 bf16
    // fp32 accumulator, M = 128; S: N = 128, both operands K-major; O: N = D, B MN-major
    const uint32_t base = (1u << 4) | (fmt << 7) | (fmt << 10) | ((128u >> 4) << 24);
    const uint32_t idesc_s = base | ((128u >> 3) << 17), idesc_o = base | (1u << 16) | (((uint32_t)D >> 3) << 17);
    const uint64_t d0 = tc_smem_desc(smem_u32(ring));
    // MN-major: 8-key groups 1024 bytes apart (the descriptor's stride), 64-column sub-tiles 16 KB apart (its leading offset)
    const uint64_t v0 = D == 64 ? d0 : d0 - (1ull << 16) + ((uint64_t)(kTcTileBytes >> 4) << 16);
    auto await = [&](unsigned long long* bar, uint32_t parity) {
        for (int i = 0; i < 64; ++i)                          // (a few microseconds of asking: try_wait answers later)
            if (at_ready(bar, parity)) return true;
        return issuer_wait(p, c, bar, parity, info.w, WHERE_RING_FULL, 2);
    };
    auto released = [&](unsigned long long* bar, uint32_t parity) { return check_phase_warp(p, c, bar, parity, info.w, WHERE_CHECK_RELEASE); };
    auto tile_of = [&](int n) { return n < 2 * both ? n & 1 : tail; };
    auto block_of = [&](int n) { return n < 2 * both ? n >> 1 : n - both; };
    // scores of the n-th block into their buffer: the block that had it before has been multiplied (its P V is ahead in the pipe)
    auto scores = [&](int n) {
        const int t = tile_of(n), j = block_of(n);
        const uint32_t k = f.tiles + (uint32_t)j, u = k & 1u, seq = first + (uint32_t)n, buf = seq % M::kScores;
        if (!await(&a->k_full[u], (k >> 1) & 1u)) return false;
        if (!(released(&a->s_full[seq % 3u], (seq / 3u) & 1u) && released(&a->k_empty[u], (k >> 1) & 1u))) return false;
        if (n == total - 1 && !released(&a->q_free, f.insts & 1u)) return false;
        tc_fence_after();
        const uint64_t qd = d0 + (uint32_t)((M::kQ + t * M::kTile) >> 4), kd = d0 + ((uint32_t)M::kK >> 4) + u * (uint32_t)(M::kTile >> 4);
        const bool alone = j >= both;                         // the other tile does not read this K tile
        if (elect_one()) {
#pragma unroll
            for (int k16 = 0; k16 < D / 16; ++k16) {
                const uint32_t off = (k16 & 3) * 2 + (k16 >> 2) * (kTcTileBytes >> 4);
                tc_mma(tmem + 128 * buf, qd + off, kd + off, idesc_s, k16 ? 1u : 0u);
            }
            tc_commit(&a->s_full[seq % 3u]);
            tc_commit(&a->k_empty[u]);
            if (alone) tc_commit(&a->k_empty[u]);
            if (n == total - 1) tc_commit(&a->q_free);        // every product that reads Q has been issued
        }
        __syncwarp();
        return true;
    };
    if (!await(&a->q_full, f.insts & 1u)) return false;
    for (int n = 0; n < (int)M::kScores && n < total; ++n)
        if (!scores(n)) return false;
    for (int n = 0; n < total; ++n) {
        const int t = tile_of(n), j = block_of(n);
        const uint32_t k = f.tiles + (uint32_t)j, u = k & 1u, buf = (first + (uint32_t)n) % M::kScores;
        if (!await(&a->p_full[t], (f.blocks[t] + (uint32_t)j) & 1u)) return false;
        if (!await(&a->v_full[u], (k >> 1) & 1u)) return false;
        // (the first P V overwrites O: the compute warps must have read the previous instruction's)
        if (j == 0 && f.outs[t] > 0 && !await(&a->o_free[t], (f.outs[t] - 1u) & 1u)) return false;
        if (!(released(&a->pv_done[t], (f.blocks[t] + (uint32_t)j) & 1u) && released(&a->v_empty[u], (k >> 1) & 1u))) return false;
        tc_fence_after();
        const uint64_t vd = v0 + ((uint32_t)M::kV >> 4) + u * (uint32_t)(M::kTile >> 4);
        const bool alone = j >= both;
        const uint32_t acc = j > 0 ? 1u : 0u;
        if (elect_one()) {
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)                  // 16 keys: 8 columns of P, 2048 bytes of V
                tc_mma_ta(tmem + M::kO + D * t, tmem + 128 * buf + 8 * k16, vd + 128 * k16, idesc_o, acc | (k16 ? 1u : 0u));
            tc_commit(&a->pv_done[t]);
            tc_commit(&a->v_empty[u]);
            if (alone) tc_commit(&a->v_empty[u]);
        }
        __syncwarp();
        if (n + (int)M::kScores < total && !scores(n + (int)M::kScores)) return false;
    }
    ++f.insts;
    f.tiles += (uint32_t)max(nbt[0], nbt[1]);
    for (int t = 0; t < 2; ++t) {
        f.blocks[t] += (uint32_t)nbt[t];
        f.outs[t] += nbt[t] > 0 ? 1u : 0u;
    }
    return true;
}

// ---- compute warps -------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void at_begin_run(Ctrl* c) {
    const int t = threadIdx.x;
    if (*(volatile uint8_t*)&c->tmem_ready == 0) {                       // (a word that only changes behind a barrier: see op_gemm_tc)
        if (t < 32) {
            __syncwarp();
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&c->tmem_base)), "r"(kTcCols)
                         : "memory");
        }
        tc_fence_before();
        compute_sync();
        tc_fence_after();
        if (t == 0) c->tmem_ready = 1;
    }
    if (t == 0) mbar_arrive(&c->attn_go);
}

// Softmax and output of one instruction.  (A wait that gives up has raised Ctrl::abort; the barrier of publish() makes that known
// to every thread.)
template <int D>
__device__ __forceinline__ void op_attention_tc(const Params& p, Ctrl* c, const mk_op_desc* op, int b, int h, int qi, int seq) {
    using M = AtMap<D>;
    constexpr float NEG_INF = -__builtin_huge_valf();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = warp >> 2, qd = warp & 3;
    const int Sq = op->i[1], Sk = op->i[2], odt = op->i[7];
    const bool causal = op->i[6] != 0, f16 = op->i[8] == DT_F16;
    const int q0 = qi * 256 + t * 128, qrow = q0 + qd * 32 + lane;         // position in the sequence
    const int kend = causal ? min(Sk, q0 + 128) : Sk;
    const int nb = at_blocks(op, qi, t);
    AttnBars* a = &c->attn;
    const uint32_t turn = (uint32_t)*(volatile uint8_t*)&c->at_turn & 1u;
    const uint32_t base = c->at_blocks[turn][t], seq0 = base + c->at_blocks[turn][t ^ 1];      // blocks of this tile, of both so far
    const int both = min(nb, at_blocks(op, qi, t ^ 1));
    if ((threadIdx.x & 127) == 0) c->at_blocks[turn ^ 1u][t] = base + (uint32_t)nb;
    phase_mark(p, c, 0);
    if (nb == 0) return;
    const uint32_t tl = *(volatile uint32_t*)&c->tmem_base + ((uint32_t)(qd * 32) << 16);
    const uint32_t ocol = tl + M::kO + D * t;
    const float sl2 = op->f[0] * kLog2e;
    float m_used = NEG_INF, l = 0.f;
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < nb; ++j) {
        const uint32_t n = seq0 + (uint32_t)at_order(t, j, both);
        const uint32_t scol = tl + 128 * (n % M::kScores);                     // the scores, and P over those already read
        ok = wait_barrier(p, c, &a->s_full[n % 3u], (n / 3u) & 1u, seq, WHERE_COMBINE, 2) && ok;
        __syncwarp();
        tc_fence_after();
        const int key0 = j * 128;
        const bool edge = key0 + 128 > kend || (causal && key0 + 128 > q0);    // a block with masked keys: those count as -inf
        const int last = causal ? min(kend - 1, qrow) : kend - 1;              // last key of this row
        float m4[4] = {NEG_INF, NEG_INF, NEG_INF, NEG_INF};
#pragma unroll 1
        for (int ch = 0; ch < 4; ++ch) {
            float s[32];
            tc_ld32(scol + ch * 32, s);
            if (edge) {
                const int n = last - (key0 + ch * 32);                         // this row's last live score of the chunk
#pragma unroll
                for (int e = 0; e < 32; ++e) s[e] = e <= n ? s[e] : NEG_INF;
            }
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
                m4[0] = max3(m4[0], s[e], s[e + 1]); m4[1] = max3(m4[1], s[e + 2], s[e + 3]);
                m4[2] = max3(m4[2], s[e + 4], s[e + 5]); m4[3] = max3(m4[3], s[e + 6], s[e + 7]);
            }
        }
        const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl2;
        // lazy rescale: keep the old maximum unless the new one is more than 2^8 above it
        float factor = 1.f;
        if (mx > m_used + kAtRescale || (m_used == NEG_INF && mx != NEG_INF)) {
            factor = m_used == NEG_INF ? 0.f : ex2(m_used - mx);
            m_used = mx;
        }
        // (for a rescale) O is complete once the previous block's P V is
        if (j > 0) ok = wait_barrier(p, c, &a->pv_done[t], (base + (uint32_t)j - 1u) & 1u, seq, WHERE_COMBINE, 2) && ok;
        __syncwarp();
        tc_fence_after();
        if (j > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
            l *= factor;
#pragma unroll 1
            for (int ch = 0; ch < D / 32; ++ch) {
                float o[32];
                tc_ld32(ocol + ch * 32, o);
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] *= factor;
                tc_st32(ocol + ch * 32, o);
            }
        }
        // P = 2^(s * scale - m), rounded to the operand type; row sum
        const float mm = m_used == NEG_INF ? 0.f : m_used;                     // (a row without a live key so far: every s is -inf)
        const float2 scale2 = make_float2(sl2, sl2), off2 = make_float2(-mm, -mm);
        float2 l4[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 1
        for (int ch = 0; ch < 4; ++ch) {
            float s[32];
            tc_ld32(scol + ch * 32, s);
            if (edge) {
                const int n = last - (key0 + ch * 32);
#pragma unroll
                for (int e = 0; e < 32; ++e) s[e] = e <= n ? s[e] : NEG_INF;   // 2^-inf = 0
            }
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
                const float2 y = fma2(make_float2(s[e], s[e + 1]), scale2, off2);
                const float2 q = make_float2(ex2(y.x), ex2(y.y));
                l4[(e >> 1) & 3] = add2(l4[(e >> 1) & 3], q);
                s[e] = q.x; s[e + 1] = q.y;
            }
            if (f16) {
#pragma unroll
                for (int e = 0; e < 16; ++e) w[e] = pack2h_fast(s[2 * e], s[2 * e + 1]);
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) w[e] = pack2(s[2 * e], s[2 * e + 1]);
            }
            tc_st16(scol + ch * 16, w);
        }
        l += ((l4[0].x + l4[0].y) + (l4[1].x + l4[1].y)) + ((l4[2].x + l4[2].y) + (l4[3].x + l4[3].y));
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && check_phase(p, c, &a->p_full[t], (base + (uint32_t)j) & 1u, seq, WHERE_CHECK_RELEASE)) mbar_arrive(&a->p_full[t]);      // S read, P written
    }
    phase_mark(p, c, 1);                                                       // last P handed over
    // ---- out = O / l ----
    ok = wait_barrier(p, c, &a->pv_done[t], (base + (uint32_t)nb - 1u) & 1u, seq, WHERE_COMBINE, 2) && ok;
    __syncwarp();
    tc_fence_after();
    const float inv = l == 0.f ? 0.f : rcp(l);
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[3]) + (((long long)b * Sq + qrow) * op->ld[3] + h * D) * 2;
#pragma unroll 1
    for (int ch = 0; ch < D / 32; ++ch) {
        float o[32];
        tc_ld32(ocol + ch * 32, o);
        if (ch == D / 32 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a->o_free[t]);
        }
        if (ok && qrow < Sq) {
#pragma unroll
            for (int e = 0; e < 32; e += 8)
                *reinterpret_cast<uint4*>(O + (ch * 32 + e) * 2) =
                    make_uint4(pack2t(odt, o[e] * inv, o[e + 1] * inv), pack2t(odt, o[e + 2] * inv, o[e + 3] * inv),
                               pack2t(odt, o[e + 4] * inv, o[e + 5] * inv), pack2t(odt, o[e + 6] * inv, o[e + 7] * inv));
        }
        __syncwarp();
    }
    phase_mark(p, c, 2);                                                       // output written
}

}  // namespace mk
