// MK_OP_GEMM on the 5th-generation tensor cores (tcgen05 + tensor memory), compute-warp side.
//   out[128 x 128 tile] = act(x @ w^T + bias) + residual        (one instruction per output tile)
//   ws += x[:, Kj] @ w[:, Kj]^T                                  (split-K partial: reduce-add)
// Same instructions, descriptor and epilogue semantics as the mma.sync body (op_gemm.cuh); the host
// library selects this body by putting the address of two tensor maps in ptr 11 (activations, then
// weights 128 bytes further: {K, rows} bf16, 128-byte swizzle, zero fill; boxes of 64 columns x 128
// rows, or x the rows there are, in whole groups of eight, for the activations of an op with fewer) and, when it has packed
// the weights into tile images, the packed array in ptr 10.
//
// Operands are K-major 128-row x 64-column tiles (16 KB).  The 128 activation rows of the m tile are
// the MMA's M side, so an accumulator row (a tensor-memory lane) is an activation row and a thread of
// the epilogue holds whole output rows: swiglu (gate columns 0..63, up columns 64..127 of the weight
// tile) pairs values of one thread.  Rows beyond M are zeros or, behind the copy's box, whatever the stage held, and never stored.
//   weights      producer warp -> eight single-tile slots in the ring's memory, across instruction
//                boundaries: they depend on nothing in the launch, so the next instruction's first
//                128 KB are already on their way while this one waits for its dependencies
//   activations  two lanes of a compute warp -> single-tile stages in the work area, after the instruction's
//                dependencies are met: 6 stages of 128 rows, or 10 of 64 rows when the op has at most
//                64.  The MMA still reads 128 rows: accumulator rows beyond the copied ones are never looked at
//                (a copy whose box has 64 rows over a tensor of 9 to 31 is slow, whatever fills the rest: gate/up of a
//                batch of 16 0.6 us per k-tile instead of 0.3; steps of 9, 16 and 31 sequences at context 1024
//                1480 -> 1098, 1431 -> 1127 and 1588 -> 1364 us with boxes of the rows there are)
//   MMA          one compute thread: 4 x tcgen05.mma (128 x 128 x 16) per k-tile; tcgen05.commit
//                returns the activation stage and the ring slot when the MMAs that read them are done
//   epilogue     all 8 compute warps; warp w reads lanes 32 (w & 3) .. +31, column half w >> 2.  Split-K partials, swiglu, accumulating
//                and plain tiles: tensor memory -> shared memory, then row-contiguous global stores / reductions from there.
//                Tiles with a residual, an activation (silu and few rows: as before) or rotated heads: straight from tensor
//                memory, a row per thread
// Every wait is bounded (wait_barrier); tensor memory is allocated by the first such instruction of a
// CTA and freed by the kernel before it exits, on every path.
#pragma once
#include "mk_device.cuh"
#include "mma.cuh"
#include "op_gemv_common.cuh"
#include "tc.cuh"

namespace mk {

// the same columns of two accumulators, `second` columns apart, added (second == 0: one accumulator)
__device__ __forceinline__ void tc_ld16_sum(uint32_t taddr, uint32_t second, float* v) {
    if (!second) { tc_ld16(taddr, v); return; }
    float w[16];
    tc_ld16x2(taddr, taddr + second, v, w);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] += w[j];
}

// Ctrl::tile_state behind an instruction of nk k-tiles: the accumulator barrier was used once more, activation stage s once more per full round
// through the stages and once more if s < nk mod stages, a weight slot per k-tile.  Thread 0 parks it during the instruction, and it becomes
// the current one behind the barrier that ends it: warps that have no part in the products may read the current one as late as that.
static_assert(kTcXHalfStages <= 10 && kTcWSlots == 8, "bits of tile_state");
__device__ __forceinline__ void tc_park_state(Ctrl* c, uint32_t state, int nk, uint32_t xstages) {
    const uint32_t full = (uint32_t)nk / xstages, rem = (uint32_t)nk - full * xstages;
    const uint32_t x = (full & 1u ? (1u << xstages) - 1u : 0u) ^ ((1u << rem) - 1u);
    c->tile_next = (uint16_t)(((state ^ x ^ 1u << 10) & 0x7ffu) | ((state >> 11) + (uint32_t)nk & 15u) << 11);
}
__device__ __forceinline__ void tc_next_state(Ctrl* c) {
    if (threadIdx.x) return;
    c->tile_state = c->tile_next;
    c->x_left[0] = c->x_left[1] = 0xff;
}

// Epilogue, second half.  The accumulator tile has been copied to shared memory (fp32, row pitch
// kTcStagePitch words); here a warp instruction covers one output row (or two half rows), four
// consecutive columns per lane, so every global access of the epilogue -- bias, residual, store or
// reduce-add -- is a contiguous 256 or 512 bytes.  Straight from tensor memory a lane holds a row,
// and a warp store touched 32 rows: measured on the lm_head tiles of batch-64 decode (rows 256 KB
// apart, lines not in L2) the stores of one tile took 9.5 us to issue.
constexpr int kTcStagePitch = 132;                          // words: conflict-free 16-byte writes by row, reads by column
static_assert(kTcXOff + 128 * kTcStagePitch * 4 <= kWorkBytes, "epilogue staging tile");
static __device__ __noinline__ void tc_write_rows(const mk_op_desc* op, const float* stage, int m0, int rows, int ncols, int col0,
                                              int n_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int odt = op->i[5], accum = op->i[6];
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]);
    const int two = ncols == 64 ? 1 : 0;                       // swiglu: 16 lanes per row, two rows per pass
    const int sub = two ? lane >> 4 : 0, c4 = (two ? lane & 15 : lane) * 4, col = col0 + c4;
    if (col >= n_out) return;
    const int step = kComputeWarps << two;
#pragma unroll 2
    for (int row = (warp << two) + sub; row < rows; row += step) {
        const float4 q = *reinterpret_cast<const float4*>(stage + row * kTcStagePitch + c4);
        const long long eo = (long long)(m0 + row) * op->ld[2] + col;
        if (accum) {
            const float f[4] = {q.x, q.y, q.z, q.w};
            red_add_bf16x4(O + eo * 2, f);
        } else if (odt == DT_F32) *reinterpret_cast<float4*>(O + eo * 4) = q;
        else *reinterpret_cast<uint2*>(O + eo * 2) = make_uint2(pack2t(odt, q.x, q.y), pack2t(odt, q.z, q.w));
    }
}

// ... of an fp32 split-K partial: nothing but the reduce-adds.
static __device__ __noinline__ void tc_reduce_rows(const mk_op_desc* op, const float* stage, int m0, int rows, int n0, int N) {
    const int warp = threadIdx.x >> 5, c4 = (threadIdx.x & 31) * 4;
    if (n0 + c4 >= N) return;
    const long long step = (long long)kComputeWarps * op->ld[2];
    float* O = reinterpret_cast<float*>(op->ptr[2]) + (long long)(m0 + warp) * op->ld[2] + n0 + c4;
    const float* from = stage + warp * kTcStagePitch + c4;
#pragma unroll 2
    for (int row = warp; row < rows; row += kComputeWarps) {
        const float4 q = *reinterpret_cast<const float4*>(from);
        red_add_f32x4(O, q.x, q.y, q.z, q.w);
        O += step;
        from += kComputeWarps * kTcStagePitch;
    }
}

// Epilogue, second half, plain tiles (not a split-K partial, not swiglu, nothing behind the bias): out = acc + bias, 128 columns.
// Specialised at compile time on the output type: with type, residual and activation as run-time switches inside the row loop the
// writer was instruction-bound (4.2 us per 128 x 128 tile against 1.3 us for the same stores, measured stand-alone).
template <int ODT>
static __device__ __noinline__ void tc_store_rows(const mk_op_desc* op, const float* stage, int m0, int rows, int col0, int n_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c4 = lane * 4, col = col0 + c4;
    if (col >= n_out) return;
    float b4[4] = {0.f, 0.f, 0.f, 0.f};
    if (const uint8_t* bias = reinterpret_cast<const uint8_t*>(op->ptr[3])) {
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(bias + (long long)col * 2));
        b4[0] = bf16_lo(w.x); b4[1] = bf16_hi(w.x); b4[2] = bf16_lo(w.y); b4[3] = bf16_hi(w.y);
    }
    const long long ldo = op->ld[2];
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)m0 * ldo + col) * (ODT == DT_F32 ? 4 : 2);
#pragma unroll 2
    for (int row = warp; row < rows; row += kComputeWarps) {
        const float4 q = *reinterpret_cast<const float4*>(stage + row * kTcStagePitch + c4);
        const float f[4] = {q.x + b4[0], q.y + b4[1], q.z + b4[2], q.w + b4[3]};
        if (ODT == DT_F32) *reinterpret_cast<float4*>(O + row * ldo * 4) = make_float4(f[0], f[1], f[2], f[3]);
        else if (ODT == DT_F16) *reinterpret_cast<uint2*>(O + row * ldo * 2) = make_uint2(pack2h(f[0], f[1]), pack2h(f[2], f[3]));
        else *reinterpret_cast<uint2*>(O + row * ldo * 2) = make_uint2(pack2(f[0], f[1]), pack2(f[2], f[3]));
    }
}
// ... of up to 32 rows with an activation from the special function units, types and activation at run time.  Straight from tensor memory two of the
// eight warps would have all of it.  9 rows of 256 columns, us per linear, from there / here: silu 7.6 / 6.9, with a residual 8.4 / 7.1, gelu
// with a residual 8.0 / 7.2 (gelu alone 6.6 from there, relu 6.6).
static __device__ __noinline__ void tc_write_few(const mk_op_desc* op, const float* stage, int rows, int col0, int n_out) {
    const int warp = threadIdx.x >> 5, c4 = (threadIdx.x & 31) * 4, col = col0 + c4, act = op->i[3], odt = op->i[5], rdt = op->i[7];
    if (col >= n_out) return;
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]);
    const uint8_t* R = reinterpret_cast<const uint8_t*>(op->ptr[4]);
    float4 r[4];                                             // (all of the warp's rows of the residual: one round trip to L2)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int row = warp + j * kComputeWarps;
        r[j] = R && row < rows ? load4_any(R, (long long)row * op->ld[4] + col, rdt) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float4 b = op->ptr[3] ? load4_any(reinterpret_cast<const uint8_t*>(op->ptr[3]), col, DT_BF16) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int row = warp + j * kComputeWarps;
        if (row >= rows) break;
        const float4 q = *reinterpret_cast<const float4*>(stage + row * kTcStagePitch + c4);
        float f[4] = {q.x + b.x, q.y + b.y, q.z + b.z, q.w + b.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = apply_act(act, f[e]);
        f[0] += r[j].x; f[1] += r[j].y; f[2] += r[j].z; f[3] += r[j].w;
        const long long eo = (long long)row * op->ld[2] + col;
        if (odt == DT_F32) *reinterpret_cast<float4*>(O + eo * 4) = make_float4(f[0], f[1], f[2], f[3]);
        else *reinterpret_cast<uint2*>(O + eo * 2) = make_uint2(pack2t(odt, f[0], f[1]), pack2t(odt, f[2], f[3]));
    }
}

// Epilogues straight from tensor memory, a row per thread and 16 columns at a time, for tiles that read another operand beside the
// accumulator or compute something from it: the row's whole piece of a residual and gate (rotated heads: the tables of the first 16
// columns) is requested before the accumulator is complete.  (A loop over few instructions: sixteen rows of a warp side by side, through the
// staging rows, are straight-line code that is fetched cold once per op.  Time from the complete accumulator, inside a prompt of 333 tokens:
// rotated heads 7.8 us, as a loop over groups of four rows 6.4, this 3.9.)
__device__ __forceinline__ bool tc_direct_wait(const Params& p, Ctrl* c, uint32_t apar, int seq) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = wait_barrier(p, c, &c->acc_full, apar, seq, WHERE_COMBINE) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    tc_fence_after();
    phase_mark(p, c, 2);                                     // accumulator complete
    __syncwarp();                                            // (the tensor-memory loads are .sync.aligned: whole warp, converged)
    return ok != 0;
}
// an activation chosen at run time on 16 values.  The common ones side by side, the others four at a time (rotated: register indices stay constant).
// us per linear of 256 columns, the writer through shared memory that had this before / all of them rotated / this: 64 rows, silu 10.6 / 13.0 / 8.1, relu
// 10.3 / 11.5 / 7.3, gelu and a residual 11.4 / 14.9 / 9.2; 200 rows, silu 14.9 / 13.1 / 8.1.
__device__ __forceinline__ void act16(int act, float* v) {
    if (act == ACT_SILU) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = apply_act(ACT_SILU, v[e]);
        return;
    }
    if (act == ACT_GELU) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = apply_act(ACT_GELU, v[e]);
        return;
    }
    if (act == ACT_RELU) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = apply_act(ACT_RELU, v[e]);
        return;
    }
    if (act == ACT_NONE) return;
#pragma unroll 1
    for (int j = 0; j < 16; j += 4) {
        float t[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = apply_act(act, v[e]);
#pragma unroll
        for (int e = 0; e < 12; ++e) v[e] = v[e + 4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[12 + e] = t[e];
    }
}
// 64 elements of a row, as many eights of them as there are, taken 16 at a time from the front
template <int DT> struct Row64 {
    static constexpr int kPer8 = DT == DT_F32 ? 2 : 1;
    uint4 w[8 * kPer8];
    __device__ __forceinline__ void load(const uint8_t* at, int cols, bool whole) {
#pragma unroll
        for (int k = 0; k < 8 * kPer8; k += 2) {
            if (kPer8 == 1 && k * 8 + 8 >= cols) {
                if (k * 8 < cols) w[k] = __ldcg(reinterpret_cast<const uint4*>(at) + k);
            } else if (k / kPer8 * 8 < cols) {
                ld32B(at + k * 16, reinterpret_cast<uint32_t*>(w + k), whole);
            }
        }
    }
    // element e of the front 16 (DT_BF16: either 16-bit type, by `f16`)
    __device__ __forceinline__ float get(int e, bool f16) const {
        const uint32_t* q = reinterpret_cast<const uint32_t*>(w);
        if (DT == DT_F32) return __uint_as_float(q[e]);
        const uint32_t x = q[e >> 1];
        if (f16) { const float2 h = unpack2h(x); return e & 1 ? h.y : h.x; }
        return e & 1 ? bf16_hi(x) : bf16_lo(x);
    }
    __device__ __forceinline__ void next() {
#pragma unroll
        for (int k = 0; k < 6 * kPer8; ++k) w[k] = w[k + 2 * kPer8];
    }
};
// 16 columns of a row as 16-bit, or the first eight of them where the row has `cols` left (whole eights; none: nothing)
template <int ODT>
__device__ __forceinline__ void put_upto16(uint8_t* at, const float* v, int cols, bool whole) {
    if (cols >= 16) put16<ODT>(at, v, whole);
    else if (cols > 0)
        *reinterpret_cast<uint4*>(at) = make_uint4(pack2t(ODT, v[0], v[1]), pack2t(ODT, v[2], v[3]), pack2t(ODT, v[4], v[5]), pack2t(ODT, v[6], v[7]));
}
// out = act(acc + bias) [* gate row of i 12 rows] [+ residual].  RKIND 0: no residual, 1: 16-bit, 2: fp32.  ACT 0: none, 1: gelu, 2: any.
// GATE: with ACT 2 decided at run time.
template <int ODT, int RKIND, int ACT, bool GATE>
static __device__ __noinline__ bool tc_cols_direct(const Params& p, Ctrl* c, const mk_op_desc* op, uint32_t two, uint32_t apar, int m0, int n0, int seq) {
    constexpr int osz = ODT == DT_F32 ? 4 : 2, rsz = RKIND == 2 ? 4 : 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, qd = warp & 3, col0 = n0 + 64 * (warp >> 2);
    const int M = op->i[0], cols = min(64, op->i[1] - col0);                     // this warp's columns
    const int row = m0 + qd * 32 + lane, safe = min(row, M - 1);
    const bool gated = GATE && op->ptr[5] != 0, r16 = op->i[7] == DT_F16, g16 = op->i[13] == DT_F16;
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)safe * op->ld[2] + col0) * osz;
    const uint8_t* R = RKIND ? reinterpret_cast<const uint8_t*>(op->ptr[4]) + ((long long)safe * op->ld[4] + col0) * rsz : nullptr;
    const uint8_t* G = gated ? reinterpret_cast<const uint8_t*>(op->ptr[5]) + ((long long)(safe / op->i[12]) * op->ld[5] + col0) * 2 : nullptr;
    const uint8_t* B = reinterpret_cast<const uint8_t*>(op->ptr[3]);
    const bool whole = ((op->ptr[2] | (uint64_t)op->ld[2] * osz) & 31) == 0;
    // (all of the row's piece: a step ahead, each step waits for a round trip to L2 -- 8.6 us for a tile with a residual)
    Row64<RKIND == 2 ? DT_F32 : DT_BF16> r;
    Row64<DT_BF16> g;
    if (RKIND) r.load(R, cols, ((op->ptr[4] | (uint64_t)op->ld[4] * rsz) & 31) == 0);
    if (gated) g.load(G, cols, ((op->ptr[5] | (uint64_t)op->ld[5] * 2) & 31) == 0);
    const bool ok = tc_direct_wait(p, c, apar, seq);
    if (!ok || m0 + qd * 32 >= M) return ok;
    const uint32_t tl = *(volatile uint32_t*)&c->tmem_base + ((uint32_t)(qd * 32) << 16) + 64 * (warp >> 2);
#pragma unroll 1
    for (int k = 0; k < cols; k += 16) {
        const bool more = k + 8 < cols;
        float v[16];
        tc_ld16_sum(tl + k, two, v);
        if (B) {                                             // (the same 16 for all lanes: one line per tile and warp)
            const uint4* at = reinterpret_cast<const uint4*>(B + (col0 + k) * 2);
            const uint4 b[2] = {__ldg(at), more ? __ldg(at + 1) : make_uint4(0u, 0u, 0u, 0u)};
            const uint32_t* q = reinterpret_cast<const uint32_t*>(b);
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] += e & 1 ? bf16_hi(q[e >> 1]) : bf16_lo(q[e >> 1]);
        }
        if (ACT == 1) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = apply_act(ACT_GELU, v[e]);
        }
        if (ACT == 2) act16(op->i[3], v);
        if (gated) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = fmaf(v[e], g.get(e, g16), RKIND ? r.get(e, r16) : 0.f);
        } else if (RKIND) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] += r.get(e, r16);
        }
        if (row < M) {
            uint8_t* at = O + k * osz;
            if (ODT == DT_F32) {
                st32B(at, reinterpret_cast<const uint32_t*>(v), whole);
                if (more) st32B(at + 32, reinterpret_cast<const uint32_t*>(v) + 8, whole);
            } else {
                put_upto16<ODT>(at, v, cols - k, whole);
            }
        }
        if (RKIND) r.next();
        if (GATE) g.next();
        __syncwarp();
    }
    return true;
}
//   rotated heads (descriptor: op_gemm.cuh): 16 columns of both halves of a head at a time, with the row's piece of the tables.  Columns behind
//   the heads (N is whole eights, not whole heads: a gate or a router packed behind v) end anywhere in a piece: it is stored as far as N goes.
template <int ODT>
static __device__ __noinline__ bool tc_rope_direct(const Params& p, Ctrl* c, const mk_op_desc* op, uint32_t two, uint32_t apar, int m0, int n0,
                                                   int seq) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, qd = warp & 3, h = warp >> 2;
    const int D = op->i[15], half = D >> 1, M = op->i[0];
    const int row = m0 + qd * 32 + lane, safe = min(row, M - 1), tok = safe % op->i[16];
    const bool t16 = op->i[17] == DT_F16;
    // D = 64: the warp's 64 columns are a head; D = 128: its share of the tile's one head is 32 columns of either half
    const int col0 = D == 64 ? 64 * h : 32 * h, d0 = D == 64 ? 0 : 32 * h;
    const bool rot = n0 + col0 < op->i[14];
    uint8_t* O = reinterpret_cast<uint8_t*>(op->ptr[2]) + ((long long)safe * op->ld[2] + n0 + col0) * 2;
    const uint8_t* C = reinterpret_cast<const uint8_t*>(op->ptr[6]) + ((long long)tok * op->ld[6] + d0) * 2;
    const uint8_t* S = reinterpret_cast<const uint8_t*>(op->ptr[7]) + ((long long)tok * op->ld[7] + d0) * 2;
    const bool whole = ((op->ptr[2] | (uint64_t)op->ld[2] * 2) & 31) == 0;
    uint4 q[8];                                              // cos of both halves, sin of both halves
    auto request = [&](int d) {
        if (rot) {
#pragma unroll
            for (int k = 0; k < 8; ++k) q[k] = __ldcg(reinterpret_cast<const uint4*>((k < 4 ? C : S) + (d + (k & 2 ? half : 0)) * 2 + (k & 1) * 16));
        }
    };
    request(0);
    const bool ok = tc_direct_wait(p, c, apar, seq);
    const int room = op->i[1] - n0 - col0;                    // columns from this warp's first to the row's end
    if (!ok || m0 + qd * 32 >= M || room <= 0) return ok;
    const uint32_t tl = *(volatile uint32_t*)&c->tmem_base + ((uint32_t)(qd * 32) << 16) + col0;
    auto get = [&](uint32_t w) { return t16 ? unpack2h(w) : make_float2(bf16_lo(w), bf16_hi(w)); };
#pragma unroll 1
    for (int d = 0; d < 32; d += 16) {
        float x1[16], x2[16];
        tc_ld16_sum(tl + d, two, x1);
        tc_ld16_sum(tl + half + d, two, x2);
        if (rot) {
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
        if (d == 0) request(16);
        if (row < M) {
            put_upto16<ODT>(O + d * 2, x1, room - d, whole);
            put_upto16<ODT>(O + (half + d) * 2, x2, room - half - d, whole);
        }
        __syncwarp();
    }
    return true;
}
// the instance of the direct epilogue for an op
template <int ODT>
__device__ __forceinline__ bool tc_direct_o(const Params& p, Ctrl* c, const mk_op_desc* op, uint32_t two, uint32_t apar, int m0, int n0, int seq) {
    if (ODT != DT_F32 && op->ptr[6]) return tc_rope_direct<ODT>(p, c, op, two, apar, m0, n0, seq);
    const int act = op->i[3];
    if (!op->ptr[4]) return act == ACT_GELU ? tc_cols_direct<ODT, 0, 1, false>(p, c, op, two, apar, m0, n0, seq) : tc_cols_direct<ODT, 0, 2, false>(p, c, op, two, apar, m0, n0, seq);
    if (op->i[7] == DT_F32) {
        if (act != ACT_NONE) return tc_cols_direct<ODT, 2, 2, true>(p, c, op, two, apar, m0, n0, seq);
        return op->ptr[5] ? tc_cols_direct<ODT, 2, 0, true>(p, c, op, two, apar, m0, n0, seq) : tc_cols_direct<ODT, 2, 0, false>(p, c, op, two, apar, m0, n0, seq);
    }
    if (act != ACT_NONE) return tc_cols_direct<ODT, 1, 2, true>(p, c, op, two, apar, m0, n0, seq);
    return op->ptr[5] ? tc_cols_direct<ODT, 1, 0, true>(p, c, op, two, apar, m0, n0, seq) : tc_cols_direct<ODT, 1, 0, false>(p, c, op, two, apar, m0, n0, seq);
}
static __device__ __noinline__ bool tc_direct(const Params& p, Ctrl* c, const mk_op_desc* op, uint32_t two, uint32_t apar, int m0, int n0, int seq) {
    const int odt = op->i[5];
    if (odt == DT_F32) return tc_direct_o<DT_F32>(p, c, op, two, apar, m0, n0, seq);
    if (odt == DT_F16) return tc_direct_o<DT_F16>(p, c, op, two, apar, m0, n0, seq);
    return tc_direct_o<DT_BF16>(p, c, op, two, apar, m0, n0, seq);
}

// Abort path: the activation tiles of an instruction that did not end have landed.  Stage s of lane s mod 2 was armed in this round if it
// lies in front of the lane's next one, else in the round before (the one before the instruction: complete).
static __device__ __noinline__ void wait_x_landed(Ctrl* c) {
    for (int lane = 0; lane < 2; ++lane) {
        const int left = c->x_left[lane], next = left & 15, stages = left & 32 ? kTcXHalfStages : kTcXStages;
        if (left == 0xff) continue;
        for (int s = lane; s < stages; s += 2)
            wait_landed(&c->x_full[s], 1, (((uint32_t)c->tile_state >> s) ^ ((uint32_t)left >> 4) ^ (s < next ? 1u : 0u)) & 1u);
    }
}

// All compute threads call this after the instruction's dependencies are met.  Returns 0, or -1
// when the CTA is aborting.
__device__ __forceinline__ int op_gemm_tc(const Params& p, Ctrl* c, uint8_t* ring, uint8_t* work, const mk_op_desc* op, int a0,
                                          int a1, int a2, int seq) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int M = op->i[0], N = op->i[1];
    const int swi = op->i[8];
    const int m0 = a0 * 128, n0 = a1 * 128;
    int kbeg, kc;
    gemm_k_range(op, a2, kbeg, kc);
    const int nk = kc / 64;
    const uint8_t* tmaps = reinterpret_cast<const uint8_t*>(op->ptr[11]);
    uint8_t* xs = work + kTcXOff;
    // activation stages: whole 128-row tiles, or twice as many 64-row half tiles
    const int xbytes = M <= 64 ? kTcTileBytes / 2 : kTcTileBytes;
    const uint32_t xcopied = (uint32_t)tc_box_rows(M) * 128u;
    const uint32_t xstages = M <= 64 ? kTcXHalfStages : kTcXStages;

    // Tensor memory is allocated by the CTA's first tile GEMM instruction and kept until the kernel
    // ends (the kernel frees it on every path); the permit to allocate is never relinquished.
    // (the test is on a word that only changes behind a barrier, so every thread takes the same branch -- not on the
    // address itself, which the allocation writes while the other warps are still arriving at the test)
    const uint32_t state = *(volatile uint16_t*)&c->tile_state;
    if (t == 0) tc_park_state(c, state, nk, xstages);
    if (*(volatile uint8_t*)&c->tmem_ready == 0) {            // (the attention op may have allocated it already)
        if (warp == 0) {
            __syncwarp();          // (.sync.aligned: the whole warp, converged)
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&c->tmem_base)), "r"(kTcCols)
                         : "memory");
        }
        tc_fence_before();
        compute_sync();
        tc_fence_after();
        if (t == 0) c->tmem_ready = 1;                          // (read again only behind the barrier that ends this instruction)
    }
    const uint32_t tmem = *(volatile uint32_t*)&c->tmem_base;
    const uint32_t apar = state >> 10 & 1u;

    phase_mark(p, c, 0);
    const uint32_t xpar0 = state & 0x3ffu, ws0 = state >> 11 & 7u, wph0 = state >> 14;
    if (warp == 2 && lane < 2) {
        // ---- activation tiles: {64 K-elements, 128 rows} at (kbeg + 64 kt, m0) ----
        // earlier instructions wrote the work area through the generic proxy (all of that is behind
        // the barrier that ended the dependency wait); the bulk copies below write it through the
        // asynchronous one, and read activations other SMs stored with plain stores
        asm volatile("fence.proxy.async;" ::: "memory");
        unsigned long long keep;
        asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(keep));
        // k-tile kt goes to stage kt mod the number of stages, each instruction starting at stage 0; the
        // parity of a stage's barriers is the one it had at the instruction's start, flipped once per
        // round through the stages (ops with 6 and with 10 stages may alternate: bit s follows barrier s)
        // (two lanes, every other k-tile each: one lane's wait / expect / copy sequence takes as long as a k-tile's MMAs)
        uint32_t s = lane, round = 1;
        for (int kt = lane; kt < nk; kt += 2) {
            if (!wait_barrier(p, c, &c->x_empty[s], ((xpar0 >> s) & 1u) ^ round, seq, WHERE_RING_EMPTY)) break;
            if (!check_phase(p, c, &c->x_full[s], ((xpar0 >> s) & 1u) ^ round ^ 1u, seq, WHERE_CHECK_ARM)) break;
            mbar_arrive_expect_tx(&c->x_full[s], xcopied);
            tma_load_2d(xs + s * xbytes, tmaps, kbeg + kt * 64, m0, &c->x_full[s], keep);
            s += 2;
            if (s >= xstages) { s -= xstages; round ^= 1u; }
        }
        c->x_left[lane] = (uint8_t)(s | round << 4 | (xstages == kTcXHalfStages ? 32u : 0u));
    } else if ((warp == 3 || warp == 1) && lane == 0) {
        // ---- MMAs: accumulator[128 activation rows][128 weight rows] += x tile . w tile^T ----
        // Two issuing threads, each with an accumulator of its own (columns 128 i ..): this one takes the
        // k-tiles kt = i, i + 2, ...; the epilogue adds the two.  What a thread executes between two
        // tcgen05.mma leaves the tensor pipe idle -- the instruction does not return before the previous
        // MMA is nearly done, so nothing is queued behind it.  Measured with a stand-alone loop: the four
        // MMAs of a k-tile take 0.19 us, the loop around them (two waits, two commits, counters) as much
        // again; a second thread's MMAs fill those gaps (0.43 -> 0.26 us per k-tile).  For the same reason
        // the loop has counters that step and wrap instead of divisions, descriptors by addition, and
        // waits that first ask with test_wait (a try_wait costs ~95 ns even on a completed phase).
        const uint32_t i = warp == 3 ? 0u : 1u;
        const uint32_t idesc = tc_idesc(op->i[9] == DT_F16);
        const uint64_t ad0 = tc_smem_desc(smem_u32(xs)), bd0 = tc_smem_desc(smem_u32(ring));
        const uint32_t xunits = (uint32_t)xbytes >> 4;                        // descriptor addresses count 16 bytes
        const uint32_t acc_at = tmem + 128 * i;
        uint32_t acc = 0, s = i, round = 0;
        uint32_t ws = ws0 + i, wph = wph0;
        if (ws >= kTcWSlots) { ws -= kTcWSlots; wph ^= 1u; }
        for (int kt = (int)i; kt < nk; kt += kTcIssuers) {
            if (!wait_barrier(p, c, &c->w_full[ws], wph, seq, WHERE_RING_FULL) ||
                !wait_barrier(p, c, &c->x_full[s], ((xpar0 >> s) & 1u) ^ round, seq, WHERE_RING_FULL))
                break;
            tc_fence_after();
            const uint64_t ad = ad0 + s * xunits, bd = bd0 + ws * (kTcTileBytes >> 4);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16) {
                tc_mma(acc_at, ad + 2 * k16, bd + 2 * k16, idesc, acc);
                acc = 1;
            }
            if (!check_phase(p, c, &c->x_empty[s], ((xpar0 >> s) & 1u) ^ round, seq, WHERE_CHECK_RELEASE) ||
                !check_phase(p, c, &c->w_empty[ws], wph, seq, WHERE_CHECK_RELEASE))
                break;
            tc_commit(&c->x_empty[s]);
            tc_commit(&c->w_empty[ws]);
            s += kTcIssuers;
            if (s >= xstages) { s -= xstages; round ^= 1u; }
            ws += kTcIssuers;
            if (ws >= kTcWSlots) { ws -= kTcWSlots; wph ^= 1u; }
        }
        tc_commit(&c->acc_full);                                            // (arrives at once when this thread had no k-tile)
        if (p.trace_cap > 0 && i == 0) c->t_phase[1] = (long long)globaltimer();     // last MMA issued
    }
    __syncwarp();

    // ---- epilogue: warp w owns lanes 32 (w & 3) .. +31 (activation rows) and column half w >> 2 ----
    const uint32_t two = nk > 1 ? 128u : 0u;                               // columns to the second issuing thread's accumulator, if it has a part
    int ok = 1;
    const bool few = M <= 32 && !op->i[6] && !swi && !op->ptr[5] && (op->i[3] == ACT_SILU || (op->i[3] == ACT_GELU && op->ptr[4]));      // tc_write_few
    if (!op->i[6] && !swi && !few && (op->ptr[6] || op->ptr[4] || op->i[3] != ACT_NONE)) {
        ok = tc_direct(p, c, op, two, apar, m0, n0, seq);
    } else {
        if (lane == 0) ok = wait_barrier(p, c, &c->acc_full, apar, seq, WHERE_COMBINE) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        tc_fence_after();
        phase_mark(p, c, 2);                                                    // accumulator complete
        __syncwarp();                                                           // (the tensor-memory loads below are .sync.aligned: whole warp, converged)
        // first half: tensor memory -> shared memory, 16 columns at a time (32 at a time needed so many registers that each call saved 320 bytes
        // per thread instead of 204, with almost no L1 to take them: 64 sequences at context 1024 1544 -> 1526 us, prompt of 333 tokens
        // 1865 -> 1845, MLP block of 256 rows 57.9 -> 56.6).  Warp w reads lanes 32 (w & 3) .. +31 (activation
        // rows) and column half w >> 2; the activation stages are free now (every MMA has completed).
        const int qd = warp & 3, h = warp >> 2;
        float* stage = reinterpret_cast<float*>(work + kTcXOff);
        const int rows = min(128, M - m0);
        if (ok && qd * 32 < rows) {
            const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
            float* srow = stage + (qd * 32 + lane) * kTcStagePitch;
            float v[16];
            if (swi) {
                // gate columns 32 h .. +31 and the up columns 64 further of the same outputs
#pragma unroll 1
                for (int ch = 0; ch < 2; ++ch) {
                    const int tcol = h * 32 + ch * 16;
                    float u[16];
                    tc_ld16_sum(tl + tcol, two, v);
                    tc_ld16_sum(tl + 64 + tcol, two, u);
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(srow + tcol + j) =
                            make_float4(v[j] * sigmoidf_(v[j]) * u[j], v[j + 1] * sigmoidf_(v[j + 1]) * u[j + 1],
                                        v[j + 2] * sigmoidf_(v[j + 2]) * u[j + 2], v[j + 3] * sigmoidf_(v[j + 3]) * u[j + 3]);
                }
            } else {
#pragma unroll 1
                for (int ch = 0; ch < 4; ++ch) {
                    const int tcol = h * 64 + ch * 16;
                    if (n0 + tcol >= N) break;
                    tc_ld16_sum(tl + tcol, two, v);
#pragma unroll
                    for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(srow + tcol + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
            }
        }
        tc_fence_before();
        compute_sync();
        if (ok) {
            if (swi) tc_write_rows(op, stage, m0, rows, 64, a1 * 64, N / 2);
            else if (op->i[6]) {                                                            // split-K partial: reduce-add
                if (op->i[5] == DT_F32) tc_reduce_rows(op, stage, m0, rows, n0, N);
                else tc_write_rows(op, stage, m0, rows, 128, n0, N);
            }
            else if (few) tc_write_few(op, stage, rows, n0, N);
            else if (op->i[5] == DT_F32) tc_store_rows<DT_F32>(op, stage, m0, rows, n0, N);
            else if (op->i[5] == DT_F16) tc_store_rows<DT_F16>(op, stage, m0, rows, n0, N);
            else tc_store_rows<DT_BF16>(op, stage, m0, rows, n0, N);
        }
    }
    tc_fence_before();
    // (no barrier: the one that publishes the instruction tells every thread of a wait that gave up, Ctrl::abort; the state and x_left then
    // stay as they are, for wait_x_landed)
    return 0;
}

}  // namespace mk
