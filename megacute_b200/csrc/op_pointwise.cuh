// Vectorised (128-bit) pointwise, norm and small decode ops.  All read and write global memory
// directly with 16-byte accesses: they are bandwidth / latency bound and need no staging.
#pragma once
#include <type_traits>
#include "mk_device.cuh"

namespace mk {

constexpr int kEwRows = 32, kEwCols = 512;                 // config.py EW_ROWS / EW_COLS

// MK_OP_FINALIZE: out = act(ws + bias) [* gate[r / i6]] + residual; ws = 0.
// ptr 0 ws (fp32), 1 out, 2 bias, 3 residual, 4 gate (or null); i 0 R, 1 C, 2 act, 3 out dtype, 4 residual dtype,
// 5 rows per instruction (schedule.py finalize_rows; 0 = kEwRows), 6 rows per gate row, 7 gate dtype
// args: 0 row tile, 1 col tile (i5 x kEwCols)
// A hop between two linears with one vector per thread: what counts is one round trip to L2 for all operands (absent ones read ws
// instead, so that no load waits for the branch of its use) and little code.  MLP block of 256 rows 55.3 -> 54.3 us, of 64 rows 37.0 -> 35.8.
static __device__ __noinline__ void op_finalize(const mk_op_desc* op, int a0, int a1) {
    const int R = op->i[0], Cc = op->i[1], act = op->i[2];
    const int tr = op->i[5] > 0 ? op->i[5] : kEwRows;
    const int r0 = a0 * tr, c0 = a1 * kEwCols;
    const int rows = min(tr, R - r0), cols = min(kEwCols, Cc - c0);
    const int vpr = cols >> 3;
    float* ws = reinterpret_cast<float*>(op->ptr[0]);
    const bool bias = op->ptr[2] != 0, res = op->ptr[3] != 0, gated = op->ptr[4] != 0;
    const int rdt = res ? op->i[4] : DT_BF16, gdt = gated ? op->i[7] : DT_BF16, group = gated ? op->i[6] : 1;
    for (int v = threadIdx.x; v < rows * vpr; v += kComputeThreads) {
        const int r = r0 + v / vpr, cidx = c0 + (v % vpr) * 8;
        const float* at = ws + (long long)r * op->ld[0] + cidx;
        const Raw8 w = load8_raw(at, 0, DT_F32);
        const uint4 b = __ldcg(bias ? reinterpret_cast<const uint4*>(op->ptr[2] + cidx * 2) : reinterpret_cast<const uint4*>(at));
        const Raw8 q = load8_raw(res ? reinterpret_cast<const void*>(op->ptr[3]) : at, res ? (long long)r * op->ld[3] + cidx : 0, rdt);
        const Raw8 g = load8_raw(gated ? reinterpret_cast<const void*>(op->ptr[4]) : at, gated ? (long long)(r / group) * op->ld[4] + cidx : 0, gdt);
        float f[8], t[8];
        unpack8_raw(w, DT_F32, f);
        unpack8(b, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += bias ? t[e] : 0.f;
        if (act != ACT_NONE) {
#pragma unroll 1
            for (int e = 0; e < 8; ++e) {                    // (rotated: register indices stay constant)
                const float y = apply_act(act, f[0]);
                f[0] = f[1]; f[1] = f[2]; f[2] = f[3]; f[3] = f[4]; f[4] = f[5]; f[5] = f[6]; f[6] = f[7]; f[7] = y;
            }
        }
        unpack8_raw(g, gdt, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= gated ? t[e] : 1.f;
        unpack8_raw(q, rdt, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += res ? t[e] : 0.f;
        store8(reinterpret_cast<void*>(op->ptr[1]), (long long)r * op->ld[1] + cidx, op->i[3], f);
        const float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        store8(ws, (long long)r * op->ld[0] + cidx, 1, z);
    }
}

// (Each instance is a function of its own: inlined into one body, the longer variants' registers and spills fell on
// the one-vector-per-thread case too, which is the norm of every decode step.)
// A row (or a lane's share of it) of at most NPER vectors per thread stays in registers between the two passes: every
// vector is requested before the first is used, and gain and bias come in pairs.  (Requested one by one,
// the vectors of a 2048-column row cost eight L2 round trips in each pass: 11 us per 8-row instruction.)
template <int NPER, bool MOD, bool X16 = false>
static __device__ __noinline__ void norm_kept(const mk_op_desc* op, int r, int first, int step, int nvec, bool live, uint8_t* work) {
    const int Cc = op->i[1], rms = op->i[2], xdt = op->i[4], odt = op->i[5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const void* X = reinterpret_cast<const void*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[1]);
    const void* W = reinterpret_cast<const void*>(op->ptr[2]);
    const void* Bv = reinterpret_cast<const void*>(op->ptr[3]);
    const void* Sc = reinterpret_cast<const void*>(op->ptr[4]);          // adaLN modulation fused in (passes.fuse_pointwise), or null
    const void* Sh = reinterpret_cast<const void*>(op->ptr[5]);
    const long long grow = live ? r / max(1, op->i[6]) : 0;
    Raw8x<X16> kr[NPER];                                  // (a 16-bit row: four registers per vector, eight vectors per lane fit)
#pragma unroll
    for (int u = 0; u < NPER; ++u) {
        const int v = first + u * step;
        if (live && v < nvec) kr[u].load(X, (long long)r * op->ld[0] + v * 8, xdt);
    }
    // gain, bias (and modulation) of the first batch are requested with the row: for a row of one vector per thread --
    // the norm of a decode step -- that is ONE L2 round trip on the instruction's critical path instead of two
    constexpr int NB = (NPER < 2 || MOD) ? 1 : 2;                  // (with the modulation's two more operands: one at a time)
    Raw8 gw[NB], bw[NB], sw[MOD ? NB : 1], tw[MOD ? NB : 1];
    auto request = [&](int u0) {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int v = first + (u0 + u) * step;
            if (live && v < nvec) {
                if (W) gw[u] = load8_raw(W, v * 8, 0);
                if (Bv) bw[u] = load8_raw(Bv, v * 8, 0);
                if (MOD) {
                    sw[u] = load8_raw(Sc, grow * op->ld[4] + v * 8, op->i[7]);
                    tw[u] = load8_raw(Sh, grow * op->ld[5] + v * 8, op->i[8]);
                }
            }
        }
    };
    request(0);
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int u = 0; u < NPER; ++u) {
        if (live && first + u * step < nvec) {
            float f[8];
            kr[u].unpack(xdt, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) { s += f[e]; ss += f[e] * f[e]; }
        }
    }
    s = warp_sum(s);
    ss = warp_sum(ss);
    float* sh = reinterpret_cast<float*>(work);
    if (lane == 0) { sh[warp * 2] = s; sh[warp * 2 + 1] = ss; }
    compute_sync();
    s = 0.f; ss = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kComputeWarps; ++w8) { s += sh[w8 * 2]; ss += sh[w8 * 2 + 1]; }
    if (!live) return;
    const float mean = rms ? 0.f : s / (float)Cc;
    const float var = ss / (float)Cc - mean * mean;
    const float rstd = rsqrt_approx(var + op->f[0]);
#pragma unroll
    for (int u0 = 0; u0 < NPER; u0 += NB) {
        if (u0 > 0) request(u0);
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            const int v = first + (u0 + u) * step;
            if (v >= nvec) continue;
            float f[8], g[8];
            kr[u0 + u].unpack(xdt, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean) * rstd;
            if (W) {
                unpack8_raw(gw[u], 0, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] *= g[e];
            }
            if (Bv) {
                unpack8_raw(bw[u], 0, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += g[e];
            }
            if (MOD) {
                float h[8];
                unpack8_raw(sw[u], op->i[7], g);
                unpack8_raw(tw[u], op->i[8], h);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = fmaf(f[e], 1.0f + g[e], h[e]);
            }
            store8(O, (long long)r * op->ld[1] + v * 8, odt, f);
        }
    }
}

// MK_OP_NORM with one row per instruction, spread over the whole CTA (i 3 = 1: ops of few rows; more rows per instruction:
// op_stream.cuh).  ptr 0 x, 1 out, 2 weight, 3 bias, 4 scale, 5 shift (adaLN modulation of the normalised row fused in:
// out = norm(x) * (1 + scale[r / group]) + shift[r / group]; or null); i 0 R, 1 C, 2 rms, 3 rows per instruction, 4 x dtype, 5 out dtype, 6 group, 7 scale dtype, 8 shift dtype; f 0 eps.
// args: 0 row tile.
// var = E[x^2] - mean^2 in fp32 (as the reference's norm kernel, megacute/ops/norm.py:94-114).
static __device__ __noinline__ void op_norm(const mk_op_desc* op, int a0, uint8_t* work) {
    const int R = op->i[0], Cc = op->i[1], rms = op->i[2], xdt = op->i[4], odt = op->i[5];
    const float eps = op->f[0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const void* X = reinterpret_cast<const void*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[1]);
    const void* W = reinterpret_cast<const void*>(op->ptr[2]);
    const void* Bv = reinterpret_cast<const void*>(op->ptr[3]);
    const int nvec = Cc >> 3;
    const int r = a0, first = threadIdx.x, step = kComputeThreads;
    const bool live = r < R;
    const int nper = (nvec + step - 1) / step;          // vectors per thread
    if (op->ptr[4] && nper <= 4) { norm_kept<4, true>(op, r, first, step, nvec, live, work); return; }
    if (nper <= 1) {
        // one vector per thread -- the norm of every decode step -- is done here, without a further call: the row's
        // vector, its gain and its bias are requested together (one L2 round trip on the instruction's critical path)
        float keep[8], gk[8], bk[8];
        float s = 0.f, ss = 0.f;
        if (live && first < nvec) {
            load8(X, (long long)r * op->ld[0] + first * 8, xdt, keep);
            if (W) load8(W, first * 8, 0, gk);
            if (Bv) load8(Bv, first * 8, 0, bk);
#pragma unroll
            for (int e = 0; e < 8; ++e) { s += keep[e]; ss += keep[e] * keep[e]; }
        }
        s = warp_sum(s);
        ss = warp_sum(ss);
        float* sh = reinterpret_cast<float*>(work);
        if (lane == 0) { sh[warp * 2] = s; sh[warp * 2 + 1] = ss; }
        compute_sync();
        s = 0.f; ss = 0.f;
#pragma unroll
        for (int w8 = 0; w8 < kComputeWarps; ++w8) { s += sh[w8 * 2]; ss += sh[w8 * 2 + 1]; }
        if (!live || first >= nvec) return;
        const float mean = rms ? 0.f : s / (float)Cc;
        const float rstd = rsqrt_approx(ss / (float)Cc - mean * mean + eps);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            keep[e] = (keep[e] - mean) * rstd;
            if (W) keep[e] *= gk[e];
            if (Bv) keep[e] += bk[e];
        }
        store8(O, (long long)r * op->ld[1] + first * 8, odt, keep);
        return;
    }
    if (nper <= 2) { norm_kept<2, false>(op, r, first, step, nvec, live, work); return; }
    if (nper <= 4) { norm_kept<4, false>(op, r, first, step, nvec, live, work); return; }
    if (nper <= 8 && xdt != DT_F32 && !op->ptr[4]) { norm_kept<8, false, true>(op, r, first, step, nvec, live, work); return; }
    // longer rows: two passes over global memory, four vectors requested at a time
    float s = 0.f, ss = 0.f;
    constexpr int UN = 4;
    if (live)
        for (int v0 = first; v0 < nvec; v0 += UN * step) {
            Raw8 rx[UN];
#pragma unroll
            for (int u = 0; u < UN; ++u)
                if (v0 + u * step < nvec) rx[u] = load8_raw(X, (long long)r * op->ld[0] + (v0 + u * step) * 8, xdt);
#pragma unroll
            for (int u = 0; u < UN; ++u) {
                if (v0 + u * step >= nvec) continue;
                float f[8];
                unpack8_raw(rx[u], xdt, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) { s += f[e]; ss += f[e] * f[e]; }
            }
        }
    s = warp_sum(s);
    ss = warp_sum(ss);
    float* sh = reinterpret_cast<float*>(work);
    if (lane == 0) { sh[warp * 2] = s; sh[warp * 2 + 1] = ss; }
    compute_sync();
    s = 0.f; ss = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kComputeWarps; ++w8) { s += sh[w8 * 2]; ss += sh[w8 * 2 + 1]; }
    if (!live) return;
    const float mean = rms ? 0.f : s / (float)Cc;
    const float var = ss / (float)Cc - mean * mean;
    const float rstd = rsqrt_approx(var + eps);
    for (int v0 = first; v0 < nvec; v0 += 2 * step) {
        Raw8 rx[2], gw[2], bw[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int v = v0 + u * step;
            if (v >= nvec) continue;
            rx[u] = load8_raw(X, (long long)r * op->ld[0] + v * 8, xdt);
            if (W) gw[u] = load8_raw(W, v * 8, 0);
            if (Bv) bw[u] = load8_raw(Bv, v * 8, 0);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int v = v0 + u * step;
            if (v >= nvec) continue;
            float f[8], g[8];
            unpack8_raw(rx[u], xdt, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean) * rstd;
            if (W) {
                unpack8_raw(gw[u], 0, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] *= g[e];
            }
            if (Bv) {
                unpack8_raw(bw[u], 0, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += g[e];
            }
            if (op->ptr[4]) {                                   // adaLN modulation fused in
                const long long grow = r / max(1, op->i[6]);
                float h[8];
                load8(reinterpret_cast<const void*>(op->ptr[4]), grow * op->ld[4] + v * 8, op->i[7], g);
                load8(reinterpret_cast<const void*>(op->ptr[5]), grow * op->ld[5] + v * 8, op->i[8], h);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = fmaf(f[e], 1.0f + g[e], h[e]);
            }
            store8(O, (long long)r * op->ld[1] + v * 8, odt, f);
        }
    }
}

// Rotate-half of one 8-wide chunk pair.  x1/x2: chunks at d and d + D/2; result rounded to bf16.
__device__ __forceinline__ void rope8(const float* x1, const float* x2, const void* cosr, const void* sinr, int d,
                                      int half, float* o1, float* o2) {
    float c1[8], c2[8], s1[8], s2[8];
    load8(cosr, d, 0, c1); load8(cosr, d + half, 0, c2);
    load8(sinr, d, 0, s1); load8(sinr, d + half, 0, s2);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        o1[e] = round_bf16(x1[e] * c1[e] - x2[e] * s1[e]);
        o2[e] = round_bf16(x2[e] * c2[e] + x1[e] * s2[e]);
    }
}

// MK_OP_ROPE_APPEND.  ptr 0 qkv, 1 cos, 2 sin, 3 pos, 4 q_out, 5 k_cache, 6 v_cache
// i 0 B, 1 H, 2 KVH, 3 D, 4 max_seq, 5 qkv dtype, 6 pos stride.  args: 0 row tile (8 sequences).
// Cache row written for sequence b: b * max_seq + pos (reference: graph.py:375-379).
static __device__ __noinline__ void op_rope_append(const mk_op_desc* op, int a0) {
    const int B = op->i[0], H = op->i[1], KVH = op->i[2], D = op->i[3], L = op->i[4], qdt = op->i[5];
    const int* posp = reinterpret_cast<const int*>(op->ptr[3]);
    const long long pstride = op->i[6];                                   // 0: one position for the batch, else one per sequence
    const int half = D >> 1, hv = half >> 3;
    const int r0 = a0 * kComputeWarps;
    const int rows = min(kComputeWarps, B - r0);
    const void* qkv = reinterpret_cast<const void*>(op->ptr[0]);
    const int units = (H + KVH) * hv;
    for (int u = threadIdx.x; u < rows * units; u += kComputeThreads) {
        const int b = r0 + u / units, rem = u % units;
        const int hh = rem / hv, d = (rem % hv) * 8;
        const int pos = posp[b * pstride];
        const __nv_bfloat16* cosr = reinterpret_cast<const __nv_bfloat16*>(op->ptr[1]) + (long long)pos * op->ld[1];
        const __nv_bfloat16* sinr = reinterpret_cast<const __nv_bfloat16*>(op->ptr[2]) + (long long)pos * op->ld[2];
        float x1[8], x2[8], o1[8], o2[8];
        load8(qkv, (long long)b * op->ld[0] + hh * D + d, qdt, x1);
        load8(qkv, (long long)b * op->ld[0] + hh * D + d + half, qdt, x2);
        rope8(x1, x2, cosr, sinr, d, half, o1, o2);
        if (hh < H) {
            store8(reinterpret_cast<void*>(op->ptr[4]), (long long)b * op->ld[4] + hh * D + d, 0, o1);
            store8(reinterpret_cast<void*>(op->ptr[4]), (long long)b * op->ld[4] + hh * D + d + half, 0, o2);
        } else {
            const long long row = (long long)b * L + pos;
            store8(reinterpret_cast<void*>(op->ptr[5]), row * op->ld[5] + (hh - H) * D + d, 0, o1);
            store8(reinterpret_cast<void*>(op->ptr[5]), row * op->ld[5] + (hh - H) * D + d + half, 0, o2);
        }
    }
    const int nv = (KVH * D) >> 3;
    for (int u = threadIdx.x; u < rows * nv; u += kComputeThreads) {
        const int b = r0 + u / nv, v = u % nv;
        float f[8];
        load8(qkv, (long long)b * op->ld[0] + (H + KVH) * D + v * 8, qdt, f);
        store8(reinterpret_cast<void*>(op->ptr[6]), ((long long)b * L + posp[b * pstride]) * op->ld[6] + v * 8, 0, f);
    }
}

// MK_OP_GATHER: out[r] = table[ids[r]] -- the embedding lookup of a decode step as the launch's first
// instructions (the reference's step calls torch.index_select before its launch,
// examples/llama/llama1b.py:103-104).  An index outside the table reads row 0.
// ptr 0 table (bf16), 1 ids (int32 column), 2 out; i 0 rows, 1 cols, 2 table rows, 3 out dtype
// args: 0 row tile (8 rows, one per warp), 1 col tile (kEwCols)
static __device__ __noinline__ void op_gather(const mk_op_desc* op, int a0, int a1, long long direct_off) {
    const int R = op->i[0], Cc = op->i[1], T = op->i[2], odt = op->i[3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r = a0 * kComputeWarps + warp;
    if (r >= R) return;
    int id = __ldcg(reinterpret_cast<const int*>(op->ptr[1]) + (long long)r * op->ld[1]);
    if (id < 0 || id >= T) id = 0;
    const int c0 = a1 * kEwCols, cols = min(kEwCols, Cc - c0);
    const void* row = reinterpret_cast<const __nv_bfloat16*>(op->ptr[0]) + (long long)id * op->ld[0];
    for (int v = lane; v < (cols >> 3); v += 32) {
        float f[8];
        load8(row, c0 + v * 8, DT_BF16, f);
        const long long e = (long long)r * op->ld[2] + c0 + v * 8;
        if (op->flags & MK_F_DIRECT_OUT) {
#pragma unroll
            for (int j = 0; j < 8; ++j) store1_direct(reinterpret_cast<float*>(op->ptr[2] + direct_off) + e + j, f[j]);
        } else {
            store8(reinterpret_cast<void*>(op->ptr[2]), e, odt, f);
        }
    }
}

// MK_OP_ARGMAX: ids[r] = argmax(x[r]), ties to the lowest index, NaN never selected -- greedy sampling as
// the launch's last instructions (the reference's step calls torch's argmax after its launch,
// examples/llama/llama1b.py:105).  A row is cut into `chunks` column ranges, one instruction each;
// every instruction leaves its best (value, index) in `part` and bumps the row's arrival count; the
// last to arrive picks the winner (one partial per thread) and resets the count.
// ptr 0 x, 1 ids (int32 column), 2 part (fp32, per row: `chunks` values, then from column ceil4(chunks) on the bits
// of their indices), 3 count
// i 0 rows, 1 cols, 2 chunks, 3 columns per chunk (multiple of 8), 4 x dtype.  args: 0 row, 1 chunk.
struct Best {
    float v;
    int i;
};
__device__ __forceinline__ Best better(Best a, Best b) {        // NaN never wins; equal values: lower index
    return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ Best warp_best(Best b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const Best other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
        b = better(b, other);
    }
    return b;
}
static __device__ __noinline__ void op_argmax(const mk_op_desc* op, int a0, int a1, Ctrl* c, uint8_t* work) {
    const int Cc = op->i[1], chunks = op->i[2], width = op->i[3], xdt = op->i[4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int r = a0, c0 = a1 * width, c1 = min(Cc, c0 + width);
    const void* X = reinterpret_cast<const void*>(op->ptr[0]);
    Best best{-__builtin_huge_valf(), 0x7fffffff};
    for (int col = c0 + t * 8; col < c1; col += kComputeThreads * 8) {
        float f[8];
        load8(X, (long long)r * op->ld[0] + col, xdt, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) best = better(best, Best{f[e], col + e});
    }
    best = warp_best(best);
    float* sv = reinterpret_cast<float*>(work);
    int* si = reinterpret_cast<int*>(work) + kComputeWarps;
    if (lane == 0) { sv[warp] = best.v; si[warp] = best.i; }
    compute_sync();
    int* ids = reinterpret_cast<int*>(op->ptr[1]) + (long long)r * op->ld[1];
    if (warp == 0) {
        best = lane < kComputeWarps ? Best{sv[lane], si[lane]} : Best{-__builtin_huge_valf(), 0x7fffffff};
        best = warp_best(best);
        if (lane == 0) {
            if (chunks == 1) {
                *ids = best.i == 0x7fffffff ? 0 : best.i;
            } else {
                float* part = reinterpret_cast<float*>(op->ptr[2]) + (long long)r * op->ld[2];
                part[a1] = best.v;
                part[((chunks + 3) & ~3) + a1] = __int_as_float(best.i);
                __threadfence();
                int* count = reinterpret_cast<int*>(op->ptr[3]) + (long long)r * op->ld[3];
                const int old = atomicAdd(count, 1);
                c->flag = (old == chunks - 1);
                if (old == chunks - 1) *count = 0;            // back to zero for the next launch
            }
        }
    }
    if (chunks == 1) return;
    compute_sync();
    if (!c->flag) return;
    __threadfence();
    const float* part = reinterpret_cast<const float*>(op->ptr[2]) + (long long)r * op->ld[2];
    best = Best{-__builtin_huge_valf(), 0x7fffffff};
    if (t < chunks) best = Best{__ldcg(part + t), __float_as_int(__ldcg(part + ((chunks + 3) & ~3) + t))};
    best = warp_best(best);
    compute_sync();                                           // sv / si of the first pass have been read
    if (lane == 0) { sv[warp] = best.v; si[warp] = best.i; }
    compute_sync();
    if (warp == 0) {
        best = lane < kComputeWarps ? Best{sv[lane], si[lane]} : Best{-__builtin_huge_valf(), 0x7fffffff};
        best = warp_best(best);
        if (lane == 0) *ids = best.i == 0x7fffffff ? 0 : best.i;
    }
}

// MK_OP_INCREMENT.  ptr 0 pos; i 0 rows of pos, 1 their stride.  One instruction.
__device__ __forceinline__ void op_increment(const mk_op_desc* op) {
    int* pos = reinterpret_cast<int*>(op->ptr[0]);
    const int rows = max(1, op->i[0]);
    for (int r = threadIdx.x; r < rows; r += kComputeThreads) pos[(long long)r * op->i[1]] += 1;
}

}  // namespace mk
