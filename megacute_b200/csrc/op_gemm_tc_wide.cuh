// MK_OP_GEMM on tcgen05 with output tiles of 256 rows (descriptor i 11 = 256) and 256 or 128 columns (i 10): linears with many rows.
//
// What bounds a tile GEMM whose operands live in L2 is the bytes an SM draws from there: measured on B200 (all 148 SMs,
// stand-alone loop) a 128 x 256 tile takes 0.46 us per 64-element k-tile of 48 KB (104 GB/s per SM) where its MMAs take
// 0.29; a 256 x 256 tile needs 64 KB for twice the flops, and a single thread that
// issues four N = 256 instructions per commit keeps the tensor pipe full (2.15 PFLOP/s with the operands in place).  So
// one instruction is a 256 x 256 tile: two 128 x 256 accumulators (rows 0..127 and 128..255: all 512 columns of tensor
// memory), three stages of 64 KB, and four roles that run ahead of one another across instruction boundaries:
//   weights      producer warp -> one 32 KB copy per k-tile (op_gemv_common.cuh), as early as a slot is free
//   activations  feeder warp (wide_feed): waits for the instruction's dependencies itself, then one bulk tensor copy of
//                256 rows x 64 columns per k-tile; rows beyond M are zero-filled
//   MMA          issuer warp, one thread (wide_issue): waits for a stage (armed once by each loader), 4 + 4 instructions, one commit.
//                It is told what to run by the feeder through Ctrl::wide_info and never touches global memory.
//   epilogue     the compute warps: warp w owns rows 32 (w & 3) .. +31 of accumulator w >> 2; it reads its 32 x 256 part in steps of
//                32 columns, each written before the next is read, and hands the accumulator back with the last one
// Tiles of 256 x 128 (kind 1; kind 0: 256 x 256) have four stages of 48 KB and half the accumulator columns.  Per k-tile, all SMs
// streaming, four tiles per SM, K from 1024 to 8192: 256 x 256 0.76 - 0.84 us, 256 x 128 0.50 - 0.56 (half a 256 x 256 tile: 0.38 -
// 0.42), 128 x 128 0.26 - 0.30 -- 128-column instructions read as many operand bytes for half the flops, and
// shared memory (128 bytes a cycle for the tensor core's reads and the copies' writes together) is what both are bound by.
// 256 x 128 is chosen where it fills the SMs better (passes.plan_tiles; its constants are fitted to measured plans, at the clocks
// of a short launch).
// The loads of the next tile therefore run through this one's epilogue, but only as far as there are stages: its MMAs wait for the
// accumulators, and those are free after seven eighths (256 x 128: three quarters) of the epilogue's arithmetic and stores.
// (With one role after the other per instruction, 128 x 256 tiles: prefill gate/up 20.5 us per 128 x 256 x 2048
// block of which 13.8 were main loop; DiT gelu tiles 28 us of which 7.)
// A run of such instructions on a CTA starts with the compute warps' arrival on gemm_go: the work area, where the
// activation slots are, belongs to other bodies before it and after the run's last accumulator.
// A body and a translation unit of its own (op_gemm_wide.cu): sharing code with the 128 x 128 body cost that one spilled registers.
#pragma once
#include "mk_device.cuh"
#include "mma.cuh"
#include "tc.cuh"

namespace mk {

// ---- feeder warp: activation tiles of one instruction (all lanes; lane 0 requests) ---------------------------------------
// `first`: the instruction before it on this CTA is not of this kind -- wait for the compute warps to turn to it.
struct WideFeed {
    uint32_t slot[2] = {0, 0}, phase[2] = {0, 0};      // position in the stages of each kind
    int kind = 0;                        // of the latest instruction
    uint32_t go = 0;                     // parity of gemm_go
    uint32_t count = 0;                  // instructions fed
};
__device__ __forceinline__ bool wide_feed(const Params& p, Ctrl* c, uint8_t* ring, const mk_op_desc* op, const Inst& in, bool first,
                                          WideFeed& f) {
    const int lane = threadIdx.x & 31;
    int kbeg, kc;
    gemm_k_range(op, in.a2, kbeg, kc);
    const int M = op->i[0], nk = kc / 64, m0 = in.a0 * 256;
    const uint8_t* tmaps = reinterpret_cast<const uint8_t*>(op->ptr[11]);
    bool ok = true;
    if (first) {
        if (lane == 0) ok = wait_barrier(p, c, &c->gemm_go, f.go, in.seq, WHERE_DEP, 2);
        f.go ^= 1u;
        if (!__all_sync(0xffffffffu, ok)) return false;
    }
    for (int k = lane; k < in.nwait; k += 32) {
        const int2 w = __ldg(p.waits + in.wait_off + k);
        ok = wait_counter(p, c, w.x, w.y, in.seq) && ok;
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    if (lane == 0) {
        // the work area was last written through the generic proxy, and so were the activations, by other SMs
        asm volatile("fence.proxy.async;" ::: "memory");
        unsigned long long keep;
        asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(keep));
        const int kind = op->i[10] == 256 ? 0 : 1;
        if (!first && kind != f.kind) {      // another division of the same memory: once the MMAs have read everything
            const int k = f.kind;
            for (uint32_t s = 0; s < (uint32_t)wide_stages(k) && ok; ++s)
                ok = wait_barrier(p, c, &c->ww_empty[k][s], (f.phase[k] ^ (s < f.slot[k] ? 1u : 0u)) ^ 1u, in.seq, WHERE_RING_EMPTY, 2);
        }
        f.kind = kind;
        uint32_t slot = f.slot[kind], phase = f.phase[kind];
        for (int kt = 0; kt < nk && ok; ++kt) {
            ok = wait_barrier(p, c, &c->ww_empty[kind][slot], phase ^ 1u, in.seq, WHERE_RING_EMPTY, 2);
            if (!ok) break;
            if (kt == 0) {
                // what the issuing thread needs to know.  Four entries: the stage just found free was filled three or four k-tiles ago,
                // so the issuing thread is done with the instruction before the four latest
                const uint32_t e = f.count & 3u;
                c->wide_info[e] = make_int4(nk, (M - m0 > 128 ? 2 : 1) | (op->i[10] >> 7) << 4, op->i[9] == DT_F16 ? 1 : 0, in.seq);
                mbar_arrive(&c->wide_told[e]);
            }
            ok = check_phase(p, c, &c->ww_full[kind][slot], phase, in.seq, WHERE_CHECK_ARM);
            if (!ok) break;
            mbar_arrive_expect_tx(&c->ww_full[kind][slot], (uint32_t)kWideXBytes);
            tma_load_2d(ring + wide_xoff((int)slot), tmaps, kbeg + kt * 64, m0, &c->ww_full[kind][slot], keep);
            if (++slot == (uint32_t)wide_stages(kind)) { slot = 0; phase ^= 1u; }
        }
        f.slot[kind] = slot;
        f.phase[kind] = phase;
    }
    ++f.count;
    return __all_sync(0xffffffffu, ok);
}
// end of the instruction list: the issuing thread leaves
__device__ __forceinline__ void wide_feed_end(Ctrl* c, const WideFeed& f) {
    if ((threadIdx.x & 31) == 0) {
        const uint32_t e = f.count & 3u;
        c->wide_info[e] = make_int4(0, 0, 0, 0);
        mbar_arrive(&c->wide_told[e]);
    }
}

// ---- issuer warp -------------------------------------------------------------------------------------------------------------
// The whole warp walks the loop and one elected lane issues: under a branch that only one lane takes, the compiler builds each
// instruction's operands in ordinary registers and moves them over one by one, and an N = 128 instruction (64 cycles of the tensor
// pipe) then takes 100 cycles to issue instead of 85 (measured stand-alone; N = 256, 128 cycles, is not affected).
__device__ __forceinline__ bool issuer_wait(const Params& p, Ctrl* c, unsigned long long* bar, uint32_t parity, int seq, int where, unsigned patience) {
    const bool ok = wait_barrier(p, c, bar, parity, seq, where, patience);
    return __all_sync(0xffffffffu, ok) != 0;
}
struct WideIssue {
    uint32_t slot[2] = {0, 0}, phase[2] = {0, 0};      // position in the stages of each kind
    uint32_t count = 0;                                 // instructions
};
// The MMAs of one instruction.  Returns false when aborting.
__device__ __forceinline__ bool wide_issue(const Params& p, Ctrl* c, uint8_t* ring, const int4& info, WideIssue& f) {
    const uint64_t d0 = tc_smem_desc(smem_u32(ring));
    const int nk = info.x;
    const uint32_t n = f.count;
    const bool both = (info.y & 15) == 2;                // rows 128..255 of the tile exist
    const uint32_t idesc = tc_idesc_n(info.z != 0, 128u * (uint32_t)(info.y >> 4));
    const uint32_t tmem = *(volatile uint32_t*)&c->tmem_base;
    const int kind = (info.y >> 4) == 2 ? 0 : 1;
    uint32_t acc = 0, s = f.slot[kind], ph = f.phase[kind];
    for (int kt = 0; kt < nk; ++kt) {
        if (!issuer_wait(p, c, &c->ww_full[kind][s], ph, info.w, WHERE_RING_FULL, 2)) return false;
        if (kt == 0) {
            if (!issuer_wait(p, c, &c->wacc_empty[0], (n & 1u) ^ 1u, info.w, WHERE_COMBINE, 2)) return false;
            // (the two halves of a 256-column tile are issued one after the other: the first may start before the second's
            // accumulator has been read)
            if (kind && !issuer_wait(p, c, &c->wacc_empty[1], (n & 1u) ^ 1u, info.w, WHERE_COMBINE, 2)) return false;
        }
        if (!check_phase_warp(p, c, &c->ww_empty[kind][s], ph, info.w, WHERE_CHECK_RELEASE)) return false;
        if (kt == nk - 1 && !(check_phase_warp(p, c, &c->wacc_full[0], n & 1u, info.w, WHERE_CHECK_RELEASE) &&
                              check_phase_warp(p, c, &c->wacc_full[1], n & 1u, info.w, WHERE_CHECK_RELEASE)))
            return false;
        tc_fence_after();
        const uint64_t ad = d0 + (uint32_t)(wide_xoff((int)s) >> 4), bd = d0 + (uint32_t)(wide_woff(kind, (int)s) >> 4);
        if (kind) {
            // N = 128: an instruction into the accumulator the previous one wrote starts late, so the two accumulators take turns
            if (elect_one()) {
                if (both) {
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) {
                        tc_mma(tmem, ad + 2 * k16, bd + 2 * k16, idesc, acc | (k16 ? 1u : 0u));
                        tc_mma(tmem + 256, ad + (kTcTileBytes >> 4) + 2 * k16, bd + 2 * k16, idesc, acc | (k16 ? 1u : 0u));
                    }
                } else {
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) tc_mma(tmem, ad + 2 * k16, bd + 2 * k16, idesc, acc | (k16 ? 1u : 0u));
                }
                if (kt == nk - 1) tc_commit(&c->wacc_full[0]);
                tc_commit(&c->ww_empty[kind][s]);
            }
        } else {
            if (elect_one()) {
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16) tc_mma(tmem, ad + 2 * k16, bd + 2 * k16, idesc, acc | (k16 ? 1u : 0u));
                if (kt == nk - 1) tc_commit(&c->wacc_full[0]);
            }
            if (kt == 0) {
                if (!issuer_wait(p, c, &c->wacc_empty[1], (n & 1u) ^ 1u, info.w, WHERE_COMBINE, 2)) return false;
                tc_fence_after();
            }
            if (elect_one()) {
                if (both) {
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16) tc_mma(tmem + 256, ad + (kTcTileBytes >> 4) + 2 * k16, bd + 2 * k16, idesc, acc | (k16 ? 1u : 0u));
                }
                tc_commit(&c->ww_empty[kind][s]);
            }
        }
        __syncwarp();
        acc = 1;
        if (++s == (uint32_t)wide_stages(kind)) { s = 0; ph ^= 1u; }
    }
    f.slot[kind] = s;
    f.phase[kind] = ph;
    if (elect_one()) {
        tc_commit(&c->wacc_full[1]);
        if (p.trace_cap > 0) c->t_phase[1] = (long long)globaltimer();
    }
    __syncwarp();
    ++f.count;
    return true;
}

// ---- compute warps: epilogue ---------------------------------------------------------------------------------------------------
// A warp's part of the tile: 32 rows (one per lane of tensor memory) x 256 columns, and 4 KB of shared memory of its own: a gate row,
// or (wide_store_any) rows of 128 bytes, 16-byte chunks swizzled by the row.
__device__ __forceinline__ uint4* wide_chunk(uint8_t* stg, int row, int ch) { return reinterpret_cast<uint4*>(stg + row * 128 + ((ch ^ (row & 7)) << 4)); }
// What an epilogue works on.
struct WideAcc {
    unsigned long long* full;            // the accumulator is complete with this parity
    unsigned long long* release;         // ... has been read
    uint32_t parity, tacc;               // tensor-memory address of the warp's lanes
    uint8_t* stg;                        // the warp's staging rows
    const uint8_t* bias;                 // the tile's 256 bias values in shared memory, or null
    int seq;
};
__device__ __forceinline__ bool wide_wait(const Params& p, Ctrl* c, const WideAcc& a) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = wait_barrier(p, c, a.full, a.parity, a.seq, WHERE_COMBINE, 2) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    tc_fence_after();
    phase_mark(p, c, 2);
    __syncwarp();                        // (the tensor-memory loads are .sync.aligned: whole warp, converged)
    return ok != 0;
}
__device__ __forceinline__ void wide_release(const Params& p, Ctrl* c, const WideAcc& a) {
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && check_phase(p, c, a.release, a.parity, a.seq, WHERE_CHECK_RELEASE)) mbar_arrive(a.release);
}
__device__ __forceinline__ void wide_bias(const uint8_t* bias, int col, float* v) {          // 32 columns from shared memory (the same for all lanes)
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        float b[8];
        unpack8(*reinterpret_cast<const uint4*>(bias + (col + j) * 2), b);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[j + e] += b[e];
    }
}

// an activation chosen at run time on 32 values: the switch outside the loop
__device__ __forceinline__ void act_all(int act, float* v) {
    if (act == ACT_RELU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
    } else if (act == ACT_SILU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = v[j] * sigmoidf_(v[j]);
    } else {
#pragma unroll 1
        for (int j = 0; j < 32; j += 8) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = apply_act(act, v[e]);
#pragma unroll
            for (int e = 0; e < 8; ++e) {                     // (rotate: register indices stay constant)
                const float t = v[e];
                v[e] = v[8 + e]; v[8 + e] = v[16 + e]; v[16 + e] = v[24 + e]; v[24 + e] = t;
            }
        }
    }
}

template <int DT>
__device__ __forceinline__ void put32(uint8_t* at, const float* v, bool whole) {
    if (DT == DT_F32) {
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(v[8 * k + e]);
            st32B(at + 32 * k, w, whole);
        }
    } else {
        put16<DT>(at, v, whole);
        put16<DT>(at + 32, v + 16, whole);
    }
}

// 16-bit outputs, no residual, 32 output columns at a time.  A loop, not 256 columns of straight-line code: fetching that code took
// longer than executing this.  ACT: 0 none, 1 gelu, 2 any (run time).
template <bool F16, bool SWI, int ACT>
__device__ __forceinline__ void wide_store16(const Params& p, Ctrl* c, const mk_op_desc* op, const WideAcc& a, int row0, int n0) {
    const int lane = threadIdx.x & 31;
    const int act = op->i[3], groups = (op->i[10] >> 5) >> (SWI ? 1 : 0);
    const bool live = row0 + lane < op->i[0];
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)(row0 + lane) * op->ld[2] + (SWI ? n0 / 2 : n0)) * 2;
    const bool whole = ((op->ptr[2] | (uint64_t)op->ld[2] * 2) & 31) == 0;
    if (!wide_wait(p, c, a)) return;
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
        float v[32];
        if (SWI) {                                           // gate columns 128 (g / 2) + 32 (g % 2) .. +31, up columns 64 further
            float u[32];
            const uint32_t tacc = a.tacc + (g >> 1) * 128 + (g & 1) * 32;
            tc_ld32(tacc, v);
            tc_ld32(tacc + 64, u);
            if (g == groups - 1) wide_release(p, c, a);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] * sigmoidf_(v[j]) * u[j];
        } else if (ACT == 1) {                               // (16 columns at a time: 32 gelus side by side are code that is fetched cold)
#pragma unroll 1
            for (int k = 0; k < 32; k += 16) {
                tc_ld16(a.tacc + g * 32 + k, v);
                if (g == groups - 1 && k) wide_release(p, c, a);
                if (a.bias) {
#pragma unroll
                    for (int j = 0; j < 16; j += 8) {
                        float b[8];
                        unpack8(*reinterpret_cast<const uint4*>(a.bias + (g * 32 + k + j) * 2), b);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[j + e] += b[e];
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = apply_act(ACT_GELU, v[j]);
                if (live) put16<F16 ? DT_F16 : DT_BF16>(O + g * 64 + k * 2, v, whole);
                __syncwarp();
            }
            continue;
        } else {
            tc_ld32(a.tacc + g * 32, v);
            if (g == groups - 1) wide_release(p, c, a);
            if (a.bias) wide_bias(a.bias, g * 32, v);
            if (ACT == 2) act_all(act, v);
        }
        if (live) put32<F16 ? DT_F16 : DT_BF16>(O + g * 64, v, whole);
        __syncwarp();
    }
}

template <int DT>
__device__ __forceinline__ void put4(uint8_t* at, const float4& o) {
    if (DT == DT_F32) *reinterpret_cast<float4*>(at) = o;
    else if (DT == DT_F16) *reinterpret_cast<uint2*>(at) = make_uint2(pack2h(o.x, o.y), pack2h(o.z, o.w));
    else *reinterpret_cast<uint2*>(at) = make_uint2(pack2(o.x, o.y), pack2(o.z, o.w));
}

// With a residual (out = acc + bias [times a gate row per i 12 rows: an adaLN-Zero block's gated residual] + residual): kDepth steps of 32
// columns of the residual are requested ahead, the first while the main loop still runs (an L2 round trip beside the operand
// stream takes 2 us).  One step per turn of the loop, the requested registers moved up: most such ops give an SM one tile, so the
// code is fetched cold, and as kDepth steps side by side that took longer than the tile (12.4 us behind the accumulator of a gated fp16 one, so 9.7: DiT of 12 images 4108 -> 3988, of 32 8114 -> 8004).
template <int RDT, int ODT, bool GATE>
__device__ __forceinline__ void wide_store_res(const Params& p, Ctrl* c, const mk_op_desc* op, const WideAcc& a, int row0, int n0) {
    constexpr int kDepth = RDT == DT_F32 ? 2 : 4, kWords = RDT == DT_F32 ? 32 : 16;
    constexpr int osz = ODT == DT_F32 ? 4 : 2, rsz = RDT == DT_F32 ? 4 : 2;
    const int lane = threadIdx.x & 31;
    const int groups = op->i[10] >> 5;
    const bool live = row0 + lane < op->i[0];
    const int row = live ? row0 + lane : op->i[0] - 1;       // (rows beyond the tensor read its last row)
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)row * op->ld[2] + n0) * osz;
    const uint8_t* R = reinterpret_cast<const uint8_t*>(op->ptr[4]) + ((long long)row * op->ld[4] + n0) * rsz;
    const bool owhole = ((op->ptr[2] | (uint64_t)op->ld[2] * osz) & 31) == 0, rwhole = ((op->ptr[4] | (uint64_t)op->ld[4] * rsz) & 31) == 0;
    uint32_t q[kDepth][kWords];
    auto request = [&](int d, int g) {                       // (steps beyond the tile read its last step)
        g = min(g, groups - 1);
#pragma unroll
        for (int k = 0; k < kWords / 8; ++k) ld32B(R + g * 32 * rsz + 32 * k, q[d] + 8 * k, rwhole);
    };
#pragma unroll
    for (int d = 0; d < kDepth; ++d) request(d, d);
    // the rest of the row comes into L2 while the main loop runs (HBM has little to do then, and much during the epilogues)
    for (int b = kDepth * 32 * rsz; b < groups * 32 * rsz; b += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(R + b) : "memory");
    if (GATE) {                                              // the gate row of the warp's rows: 256 columns as fp32 in its staging rows
        const uint8_t* G = reinterpret_cast<const uint8_t*>(op->ptr[5]) + ((long long)(row0 / op->i[12]) * op->ld[5] + n0) * 2;
        if (lane < groups * 4) {
            float gt[8];
            load8(G, lane * 8, op->i[13], gt);
            float4* to = reinterpret_cast<float4*>(a.stg) + lane * 2;
            to[0] = make_float4(gt[0], gt[1], gt[2], gt[3]);
            to[1] = make_float4(gt[4], gt[5], gt[6], gt[7]);
        }
        __syncwarp();
    }
    if (!wide_wait(p, c, a)) return;
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
        float v[32];
        tc_ld32(a.tacc + g * 32, v);
        if (g == groups - 1) wide_release(p, c, a);
        if (a.bias) wide_bias(a.bias, g * 32, v);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            float4 gt = make_float4(1.f, 1.f, 1.f, 1.f);
            if (GATE) gt = reinterpret_cast<const float4*>(a.stg)[g * 8 + j / 4];
            float f[4];
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                if (RDT == DT_F32) { f[e] = __uint_as_float(q[0][(j + e) % kWords]); f[e + 1] = __uint_as_float(q[0][(j + e + 1) % kWords]); }
                else if (RDT == DT_F16) { const float2 x = unpack2h(q[0][(j + e) / 2]); f[e] = x.x; f[e + 1] = x.y; }
                else { f[e] = bf16_lo(q[0][(j + e) / 2]); f[e + 1] = bf16_hi(q[0][(j + e) / 2]); }
            }
            v[j] = GATE ? fmaf(v[j], gt.x, f[0]) : v[j] + f[0];
            v[j + 1] = GATE ? fmaf(v[j + 1], gt.y, f[1]) : v[j + 1] + f[1];
            v[j + 2] = GATE ? fmaf(v[j + 2], gt.z, f[2]) : v[j + 2] + f[2];
            v[j + 3] = GATE ? fmaf(v[j + 3], gt.w, f[3]) : v[j + 3] + f[3];
        }
#pragma unroll
        for (int d = 0; d + 1 < kDepth; ++d)
#pragma unroll
            for (int k = 0; k < kWords; ++k) q[d][k] = q[d + 1][k];
        request(kDepth - 1, g + kDepth);
        if (live) put32<ODT>(O + g * 32 * osz, v, owhole);
        __syncwarp();
    }
}

// 16-bit outputs whose first i 14 columns are heads (i 15 = 64 or 128 columns each) to be rotated: row r by row r mod i 16 of the 16-bit
// cos and sin tables (ptr 6, 7).  16 columns of both halves of a head at a time, for all heads of the tile, so that a thread
// reads its table row once per tile (64 KB beside 128 KB of output; once per head it would be 256).  The first such piece of
// the tables is requested into registers while the main loop runs, the one after the current into the thread's 128 bytes of the
// warp's staging rows (a second set of registers spills).
template <bool F16, bool T16>
__device__ __forceinline__ void wide_store_rope(const Params& p, Ctrl* c, const mk_op_desc* op, const WideAcc& a, int row0, int n0) {
    constexpr int ODT = F16 ? DT_F16 : DT_BF16;
    const int lane = threadIdx.x & 31;
    const int cols = op->i[10], D = op->i[15], half = D >> 1, rot = op->i[14] - n0;
    const bool live = row0 + lane < op->i[0];
    const int row = live ? row0 + lane : op->i[0] - 1, tok = row % op->i[16];
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)row * op->ld[2] + n0) * 2;
    const uint8_t* C = reinterpret_cast<const uint8_t*>(op->ptr[6]) + (long long)tok * op->ld[6] * 2;
    const uint8_t* S = reinterpret_cast<const uint8_t*>(op->ptr[7]) + (long long)tok * op->ld[7] * 2;
    const bool whole = ((op->ptr[2] | (uint64_t)op->ld[2] * 2) & 31) == 0;
    uint4 q[8];                                              // cos of both halves, sin of both halves
    auto from = [&](int k, int d) { return (k < 4 ? C : S) + (d + (k & 2 ? half : 0)) * 2 + (k & 1) * 16; };
    auto next = [&](int d) {
        if (d < half && rot > 0)
#pragma unroll
            for (int k = 0; k < 8; ++k) cp_async16(wide_chunk(a.stg, lane, k), from(k, d), true);
        cp_async_commit();
    };
    auto get = [&](uint32_t w) { return T16 ? unpack2h(w) : make_float2(bf16_lo(w), bf16_hi(w)); };
    if (rot > 0)
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = __ldcg(reinterpret_cast<const uint4*>(from(k, 0)));
    next(16);
    if (!wide_wait(p, c, a)) return;
#pragma unroll 1
    for (int d = 0;;) {
#pragma unroll 1
        for (int h = 0; h < cols; h += D) {
            float x1[16], x2[16];
            __syncwarp();
            tc_ld16x2(a.tacc + h + d, a.tacc + h + half + d, x1, x2);
            if (d + 16 == half && h + D == cols) wide_release(p, c, a);
            if (h < rot) {
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const uint32_t* t = reinterpret_cast<const uint32_t*>(q);
                    const float2 c1 = get(t[e / 2]), c2 = get(t[8 + e / 2]), s1 = get(t[16 + e / 2]), s2 = get(t[24 + e / 2]);
                    const float u0 = x1[e], v0 = x2[e], u1 = x1[e + 1], v1 = x2[e + 1];
                    x1[e] = u0 * c1.x - v0 * s1.x;
                    x2[e] = v0 * c2.x + u0 * s2.x;
                    x1[e + 1] = u1 * c1.y - v1 * s1.y;
                    x2[e + 1] = v1 * c2.y + u1 * s2.y;
                }
            }
            if (live) {
                put16<ODT>(O + (h + d) * 2, x1, whole);
                put16<ODT>(O + (h + half + d) * 2, x2, whole);
            }
        }
        d += 16;
        if (d >= half) break;
        asm volatile("cp.async.wait_all;" ::: "memory");     // (the thread's own copies)
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = *wide_chunk(a.stg, lane, k);
        next(d + 16);
    }
    __syncwarp();
}

// Everything else -- fp32 output, split-K partial (reduce-add), an activation in front of a residual: the same without requests ahead.
__device__ __forceinline__ void wide_store_any(const Params& p, Ctrl* c, const mk_op_desc* op, const WideAcc& a, int row0, int n0) {
    const int lane = threadIdx.x & 31;
    const int act = op->i[3], odt = op->i[5], rdt = op->i[7];
    const bool accum = op->i[6] != 0, swi = op->i[8] != 0;
    const int groups = (op->i[10] >> 5) >> (swi ? 1 : 0);
    const int rows = min(32, op->i[0] - row0);
    const int r = lane >> 3, c4 = (lane & 7) * 4, osz = odt == DT_F32 ? 4 : 2;
    const long long ldo = (long long)op->ld[2] * osz;
    const int col0 = (swi ? n0 / 2 : n0) + c4;
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + (long long)(row0 + r) * ldo + col0 * osz;
    const uint8_t* R = accum ? nullptr : reinterpret_cast<const uint8_t*>(op->ptr[4]);
    const uint8_t* G = accum ? nullptr : reinterpret_cast<const uint8_t*>(op->ptr[5]);
    if (!wide_wait(p, c, a)) return;
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
        float v[32];
        if (swi) {
            float u[32];
            tc_ld32(a.tacc + (g >> 1) * 128 + (g & 1) * 32, v);
            tc_ld32(a.tacc + (g >> 1) * 128 + 64 + (g & 1) * 32, u);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] * sigmoidf_(v[j]) * u[j];
        } else {
            tc_ld32(a.tacc + g * 32, v);
            if (a.bias) wide_bias(a.bias, g * 32, v);
            if (act != ACT_NONE) act_all(act, v);
        }
        if (g == groups - 1) wide_release(p, c, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(wide_chunk(a.stg, lane, j)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
            if (j * 4 + r >= rows) break;
            float4 o = *reinterpret_cast<const float4*>(wide_chunk(a.stg, j * 4 + r, lane & 7));
            if (G) {
                const float4 f = load4_any(G, (long long)((row0 + j * 4 + r) / op->i[12]) * op->ld[5] + col0 + g * 32, op->i[13]);
                o.x *= f.x; o.y *= f.y; o.z *= f.z; o.w *= f.w;
            }
            if (R) {
                const float4 f = load4_any(R, (long long)(row0 + j * 4 + r) * op->ld[4] + col0 + g * 32, rdt);
                o.x += f.x; o.y += f.y; o.z += f.z; o.w += f.w;
            }
            uint8_t* at = O + (long long)(j * 4) * ldo + g * 32 * osz;
            if (accum) {
                if (odt == DT_F32) red_add_f32x4(reinterpret_cast<float*>(at), o.x, o.y, o.z, o.w);
                else red_add_bf16x4(at, &o.x);
            } else if (odt == DT_F32) put4<DT_F32>(at, o);
            else if (odt == DT_F16) put4<DT_F16>(at, o);
            else put4<DT_BF16>(at, o);
        }
        __syncwarp();
    }
}

// The epilogue of an op, chosen once per run of instructions: each has a function of its own around it (op_gemm_wide.cu) and so a
// register allocation of its own -- called per instruction they pay ~60 saved and restored registers each time, inlined
// side by side they spill, and with the shared memory taken every such access is an L2 round trip behind the operand stream.
// WIDE_PLAIN .. WIDE_ROPE_T16 (fp16 tables): + 16 for fp16 output.  WIDE_RES: + residual dtype | output dtype << 2 | gate << 4.
enum { WIDE_PLAIN = 0, WIDE_SWIGLU, WIDE_GELU, WIDE_ACT, WIDE_ANY, WIDE_ROPE, WIDE_ROPE_T16, WIDE_RES = 32 };
__device__ __forceinline__ int wide_variant(const mk_op_desc* op) {
    const int odt = op->i[5];
    if (op->i[6]) return WIDE_ANY;
    const bool gate32 = !op->ptr[5] || (op->i[12] % 32 == 0 && op->i[13] != DT_F32);         // a warp's 32 rows share a 16-bit gate row
    if (op->ptr[4]) return op->i[3] == ACT_NONE && !op->i[8] && gate32 ? WIDE_RES + (op->i[7] | odt << 2 | (op->ptr[5] ? 16 : 0)) : WIDE_ANY;
    if (odt == DT_F32) return WIDE_ANY;
    if (op->ptr[6]) return (op->i[17] == DT_F16 ? WIDE_ROPE_T16 : WIDE_ROPE) + (odt == DT_F16 ? 16 : 0);
    const int v = op->i[8] ? WIDE_SWIGLU : op->i[3] == ACT_NONE ? WIDE_PLAIN : op->i[3] == ACT_GELU ? WIDE_GELU : WIDE_ACT;
    return v + (odt == DT_F16 ? 16 : 0);
}

// Before the first instruction of a run: tensor memory (allocated by the CTA's first tcgen05 instruction and kept until the
// kernel ends; the branch is taken on a word that only changes behind a barrier, see op_gemm_tc), then the go for the feeder.
__device__ __forceinline__ void wide_begin_run(Ctrl* c) {
    const int t = threadIdx.x;
    if (*(volatile uint8_t*)&c->tmem_ready == 0) {
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
    if (t == 0) mbar_arrive(&c->gemm_go);
}

// Epilogue of one instruction; all compute threads.  (A wait that gives up has raised Ctrl::abort; the barrier of publish()
// makes that known to every thread.)
template <int V>
__device__ __forceinline__ void op_gemm_tc_wide(const Params& p, Ctrl* c, uint8_t* ring, const mk_op_desc* op, int a0, int a1, int seq) {
    const int t = threadIdx.x, warp = t >> 5;
    const int qd = warp & 3, h = warp >> 2;
    const uint32_t par = *(volatile uint32_t*)&c->wide_uses & 1u;
    const int n0 = a1 * op->i[10], row0 = a0 * 256 + h * 128 + qd * 32;
    phase_mark(p, c, 0);
    const uint8_t* bias = nullptr;
    if (op->ptr[3] && !op->i[6] && !op->i[8]) {                 // (behind the barrier that ended the previous instruction)
        uint8_t* bs = ring + kWideBiasOff;
        if (t < op->i[10] / 8) reinterpret_cast<uint4*>(bs)[t] = __ldg(reinterpret_cast<const uint4*>(op->ptr[3] + (uint64_t)n0 * 2) + t);
        compute_sync();
        bias = bs;
    }
    const WideAcc a{&c->wacc_full[h], &c->wacc_empty[h], par, *(volatile uint32_t*)&c->tmem_base + ((uint32_t)(qd * 32) << 16) + 256u * h,
                    ring + kWideStageOff + warp * 4096, bias, seq};
    if (row0 >= op->i[0]) {                                     // (rows beyond M)
        if (wide_wait(p, c, a)) wide_release(p, c, a);
        return;
    }
    if constexpr (V >= WIDE_RES) {
        wide_store_res<V & 3, (V >> 2) & 3, (V & 16) != 0>(p, c, op, a, row0, n0);
    } else {
        constexpr bool f16 = (V & 16) != 0;
        constexpr int kind = V & 15;
        if constexpr (kind == WIDE_PLAIN) wide_store16<f16, false, 0>(p, c, op, a, row0, n0);
        else if constexpr (kind == WIDE_SWIGLU) wide_store16<f16, true, 0>(p, c, op, a, row0, n0);
        else if constexpr (kind == WIDE_GELU) wide_store16<f16, false, 1>(p, c, op, a, row0, n0);
        else if constexpr (kind == WIDE_ROPE || kind == WIDE_ROPE_T16) wide_store_rope<f16, kind == WIDE_ROPE_T16>(p, c, op, a, row0, n0);
        else if constexpr (kind == WIDE_ACT) wide_store16<f16, false, 2>(p, c, op, a, row0, n0);
        else wide_store_any(p, c, op, a, row0, n0);
    }
}

}  // namespace mk
