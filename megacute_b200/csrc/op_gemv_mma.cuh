// Compute-warp side of the tensor-core streaming linear (MK_OP_GEMV with GEMV_F_UNITS):
//   out[m][o] = act(rstd[m] * sum_k w[o][k] * (x[m][k] * gain[k]) + bias[o]) + residual[m][o],  m < M <= 8
// Stage layout, flag and producer side: op_gemv_common.cuh.
//
// The code is deliberately compact (rolled outer loops, one code path for every K): a decode step
// runs each op body once per instruction, so the bodies execute cold and a large unrolled body is
// paid for in instruction-cache misses (measured: "no instruction" was the top stall reason).
//
// Shared memory (work region):
//   xf       [M][K/16][4 lanes][4 words]: x * gain split into bf16 high and low parts, stored in
//            MMA B-fragment order: for k-step s and lane quad position j the 16 bytes are
//            {hi k=2j,2j+1 | hi k=2j+8,2j+9 | lo k=2j,2j+1 | lo k=2j+8,2j+9} of the 16 k of step s,
//            so a lane fetches its whole B operand of a k-step with one 128-bit load.  Rows are
//            padded by 64 bytes so the 8 activation rows of a quarter-warp hit different banks.
//   red      [4 slots][8 warps][32 lanes] float4: per-warp partial 16 x 8 tiles of a row group
//   rowstat  [8 warps][8 rows] partial sums of x^2
//
// The eight compute warps only stream: each deposits its partial tile of a row group in a slot and
// moves on to the next stage.  A ninth warp, the finisher (gemv_finisher below), adds the eight
// partials and runs the epilogue (rstd, bias, activation, swiglu, residual, store).  With the
// epilogue on a compute warp that warp is late for the next group by the epilogue's length, and
// since every group needs every warp's K slice each group costs MMA + combine + epilogue; the ring
// has only two stages, so a stage's period is (that + the refill latency) / 2.
// Hand-over per slot: Ctrl::slot_full (8 arrivals, one per compute warp) and Ctrl::slot_free (the
// finisher); Ctrl::epi_done tells the compute warps that the instruction's last store has left.
#pragma once
#include "mma.cuh"
#include "op_gemv_common.cuh"

namespace mk {

constexpr int kMmaRedOff = 66 * 1024;                      // xf takes at most 64 KB + 512 B
constexpr int kMmaStatOff = kMmaRedOff + 4 * 8 * 32 * 16;  // + 16 KB

__device__ __forceinline__ float4 lds_volatile4(const float4* p) {
    float4 v;
    asm volatile("ld.volatile.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(p)) : "memory");
    return v;
}
__device__ __forceinline__ void sts_volatile4(float4* p, float4 v) {
    asm volatile("st.volatile.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(smem_u32(p)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// The op waits for its own dependencies so that loads which depend on nothing in the launch (the
// norm gain) are already in flight when the wait ends.
// DIRECT: x is a direct operand (mk_device.cuh).  A function of its own, so that neither form runs the other's code.
template <bool DIRECT>
__device__ __forceinline__ void gemv_mma(const Params& p, Ctrl* c, uint8_t* ring, uint8_t* work, const mk_op_desc* op,
                                         int o0, int o1, int seq, RingPos& pos, int nwait, int wait_off) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int M = op->i[0], K = op->i[2];
    const bool swi = op->flags & GEMV_F_SWIGLU, rms = op->flags & GEMV_F_RMS;
    const int S = (K + kSegElems - 1) / kSegElems;
    const int xrow = K * 4 + 64;                                              // bytes per activation row of xf
    uint8_t* xf = work;
    float4* red = reinterpret_cast<float4*>(work + kMmaRedOff);
    float* rowstat = reinterpret_cast<float*>(work + kMmaStatOff);

    // ---- before the dependency wait: the norm gain of this thread's first vector ----
    const int nv = K >> 3;
    const uint4* gain = (rms && op->ptr[5]) ? reinterpret_cast<const uint4*>(op->ptr[5]) : nullptr;
    const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    const uint4 g0 = gain && t < nv ? __ldg(gain + t) : ones;
    // everything below that does not depend on the activations is also set up before the wait:
    // the op runs once per instruction, cold, and this code would otherwise sit between the
    // arrival of x and the first MMA
    const int n = o1 - o0;
    const int ngroups = (swi ? 2 : 1) * ((n + 15) / 16);
    constexpr int kSlice = kSegElems / kComputeWarps;                         // 256: a warp's K slice of a segment
    const int kw = warp * kSlice;
    // B operand (16 k x 8 columns).  Up to 4 activation rows: columns 0..3 carry the high parts of
    // rows 0..3 and columns 4..7 their low parts, so ONE MMA per k-step yields both products (they
    // are added in the epilogue).  5 to 8 rows: a column per row, high and low parts in two MMAs.
    const bool packed = M <= 4;
    const int bn = lane >> 2;                                                 // this lane's B column
    const int bm = packed ? (bn & 3) : bn;                                    // the activation row behind it
    const uint32_t a_lane = (uint32_t)((lane & 15) * kSegStride + ((lane >> 4) * 8) * 2 + kw * 2);
    const uint32_t b_lane = smem_u32(xf) + (bm < M ? bm : 0) * xrow + (kw >> 4) * 64 + (lane & 3) * 16 +
                            (packed ? (bn >> 2) * 8 : 0);
    const int xdt = op->i[4];
    const void* x = reinterpret_cast<const void*>(op->ptr[0] + (DIRECT ? p.direct_off : 0));
    const long long ldx = op->ld[0];
    if (wait_deps(p, c, DIRECT ? 0 : nwait, wait_off, seq)) return;
    if (t == 0) {
        mbar_arrive(&c->deps_met);          // the finisher may now read the residual of the first row group
        if (p.trace_cap > 0) c->t_dep = (long long)globaltimer();
    }

    // ---- stage x * gain (high + low bf16 parts, fragment order); accumulate sum(x^2) per row ----
    // (one vector of a row at a time here, four k-steps at a time below: what counts is that the body has few registers.  With four
    // vectors and eight k-steps it saved and restored 43 callee-saved registers per call, 44 KB of local memory each way through a
    // path of 32 bytes a cycle: batch 1 at context 1024 852 -> 831 us, at 16384 985 -> 970, five sequences 1172 -> 1137, an MLP block of
    // one row 28.1 -> 27.0.  With two k-steps batch 1 is back at 844.)
    if (M == 1 || xdt != DT_F32 || (K & 255) != 0) {
#pragma unroll 1
        for (int m = 0; m < M; ++m) {
            float ss = 0.f;
#pragma unroll 1
            for (int v = t; v < nv; v += kComputeThreads) {
                float f[8], gq[8];
                if (DIRECT) {
                    const float* at = reinterpret_cast<const float*>(x) + m * ldx + v * 8;
                    DirectWait w;
                    while (load8_direct(at, f) == kUnwritten)
                        if (!w.again(p, c)) { c->flag = -1 - seq; break; }
                } else {
                    load8(x, m * ldx + v * 8, xdt, f);
                }
                unpack8(v == t ? g0 : (gain ? __ldg(gain + v) : ones), gq);
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float y0 = f[2 * j] * gq[2 * j], y1 = f[2 * j + 1] * gq[2 * j + 1];
                    ss += f[2 * j] * f[2 * j] + f[2 * j + 1] * f[2 * j + 1];
                    const float h0 = round_bf16(y0), h1 = round_bf16(y1);
                    hi[j] = pack2(h0, h1);
                    lo[j] = pack2(y0 - h0, y1 - h1);
                }
                uint32_t* d = reinterpret_cast<uint32_t*>(xf + m * xrow + (v >> 1) * 64 + (v & 1) * 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) { d[j * 4] = hi[j]; d[j * 4 + 2] = lo[j]; }
            }
            if (rms) {
                ss = warp_sum(ss);
                if (lane == 0) rowstat[warp * 8 + m] = ss;
            }
        }
        compute_sync();
    } else {
        // Two rows and more.  One vector of a row at a time, as above, a row takes 0.65 us: a round trip to L2 and then as long a chain of
        // conversions, word-wise stores and the sum's shuffles, with two warps per scheduler.  Here all rows are on their way at once, as
        // copies into the place of their own fragments (8 elements take 32 bytes either way), without registers; then a lane makes the
        // 16-byte fragments of its k-steps, 2 + 2 elements each, of two rows side by side (the last row of an odd number twice, with
        // the same result).  Five rows of 2048 3.4 -> 2.1 us, eight 5.4 -> 2.9.  Direct operands are looked at in registers, two rows at a time.
        if (!DIRECT) {
#pragma unroll 1
            for (int m = 0; m < M; ++m) {
#pragma unroll 1
                for (int v = t; v < nv; v += kComputeThreads) {
                    const float* from = reinterpret_cast<const float*>(x) + m * ldx + v * 8;
                    uint8_t* to = xf + m * xrow + v * 32;
                    cp_async16(to, from, true);
                    cp_async16(to + 16, from + 4, true);
                }
            }
        }
        // the k-steps of the vectors that this warp has copied: 16 of every 128
        constexpr int kBlocks = DIRECT ? 1 : 2;
        const int nb = K >> 4, u1 = warp * 8 * kBlocks + (lane >> 2), j = lane & 3;
        auto gain2 = [&](int u, int h) { return gain ? __ldg(reinterpret_cast<const uint32_t*>(gain) + u * 8 + j + 4 * h) : 0x3f803f80u; };
        uint32_t g1[kBlocks][2] = {};
        if (!DIRECT && u1 < nb) {
#pragma unroll
            for (int q = 0; q < kBlocks; ++q) { g1[q][0] = gain2(u1 + 8 * q, 0); g1[q][1] = gain2(u1 + 8 * q, 1); }
        }
        if (!DIRECT) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
        }
#pragma unroll 1
        for (int m = 0; m < M; m += 2) {
            const int m2 = min(m + 1, M - 1);
            float s0 = 0.f, s1 = 0.f;
            const uint32_t at = smem_u32(xf) + m * xrow + j * 16, next = m2 > m ? xrow : 0;
#pragma unroll 1
            for (int u = u1; u < nb; u += 64 * kBlocks) {
                const uint32_t to = at + u * 64;
                uint2 w[2][kBlocks][2];
                uint32_t g[kBlocks][2];
#pragma unroll
                for (int q = 0; q < kBlocks; ++q) { g[q][0] = g1[q][0]; g[q][1] = g1[q][1]; }
                if (DIRECT || u != u1) {
#pragma unroll
                    for (int q = 0; q < kBlocks; ++q) { g[q][0] = gain2(u + 8 * q, 0); g[q][1] = gain2(u + 8 * q, 1); }
                }
                if (DIRECT) {
                    const float* from = reinterpret_cast<const float*>(x) + m * ldx + u * 16 + j * 2;
#pragma unroll 1
                    for (DirectWait dw;;) {
                        uint32_t most = 0;
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int q = 0; q < kBlocks; ++q)
#pragma unroll
                                for (int h = 0; h < 2; ++h) w[r][q][h] = load2_direct(from + (r && m2 > m ? ldx : 0) + q * 128 + h * 8);
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int q = 0; q < kBlocks; ++q)
#pragma unroll
                                for (int h = 0; h < 2; ++h) most = max(most, max(w[r][q][h].x, w[r][q][h].y));
                        if (most != kUnwritten) break;
                        if (!dw.again(p, c)) { c->flag = -1 - seq; break; }
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < kBlocks; ++q)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            w[0][q][h] = lds64(to - j * 8 + q * 512 + h * 32);
                            w[1][q][h] = lds64(to - j * 8 + q * 512 + h * 32 + next);
                        }
                }
                if (!DIRECT) __syncwarp();                                   // (the lanes of a k-step have read its 64 bytes)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int q = 0; q < kBlocks; ++q) {
                        uint32_t hi[2], lo[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float vx = __uint_as_float(w[r][q][h].x), vy = __uint_as_float(w[r][q][h].y);
                            const float y0 = vx * bf16_lo(g[q][h]), y1 = vy * bf16_hi(g[q][h]);
                            if (r) s1 += vx * vx + vy * vy;
                            else s0 += vx * vx + vy * vy;
                            hi[h] = pack2(y0, y1);
                            lo[h] = pack2(y0 - bf16_lo(hi[h]), y1 - bf16_hi(hi[h]));
                        }
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + q * 512 + r * next), "r"(hi[0]), "r"(hi[1]), "r"(lo[0]), "r"(lo[1])
                                     : "memory");
                    }
            }
            if (rms) {                                                       // both rows' sums: the lower half warp takes the first row's
                const bool up = lane & 16;
                float ss = (up ? s1 : s0) + __shfl_xor_sync(0xffffffffu, up ? s0 : s1, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                if ((lane & 15) == 0) rowstat[warp * 8 + (up ? m2 : m)] = ss;
            }
        }
        compute_sync();
    }
    phase_mark(p, c, 0);
#pragma unroll 1
    for (int g = 0; g < ngroups; ++g) {
        // four independent accumulator tiles (even / odd k-step x high / low part of x) keep the
        // chain of dependent MMAs short; they are summed once per row group
        float accs[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) accs[q][e] = 0.f;
        bool ok = true;
#pragma unroll 1
        for (int seg = 0; seg < S; ++seg) {
            ok = wait_barrier(p, c, &c->full[pos.stage], pos.phase, seq, WHERE_RING_FULL) && ok;
            if (g == 0 && seg == 0) phase_mark(p, c, 1);
            int left = min(kSegElems, K - seg * kSegElems) - kw;              // K elements of this warp's slice
            if (ok) {
                uint32_t a_base = smem_u32(ring + pos.stage * kStageBytes) + a_lane;
                uint32_t b_base = b_lane + seg * (kSegElems / 16) * 64;
                // batches of four k-steps without a test inside (with one per step: batch 1 757 us instead of 739, five sequences 1129
                // instead of 1118, an MLP block of one row 27.1 instead of 25.4), then what is left of a slice one by one.  Lanes of absent
                // activation rows feed zeros and stay out of the load: with one row only a quarter of the warp touches shared memory
                left = min(left, kSlice);
#pragma unroll 1
                for (; left > 0; left -= 64) {
                    const int steps = left >= 64 ? 4 : left >> 4;
                    if (steps < 4) {
#pragma unroll 1
                        for (int ks = 0; ks < steps; ++ks) {
                            uint32_t a[4];
                            ldmatrix_x4(a_base + ks * 32, a[0], a[1], a[2], a[3]);
                            if (packed) {
                                const uint2 b = bm < M ? lds64(b_base + ks * 64) : make_uint2(0u, 0u);
                                mma_bf16(accs[0], a, b.x, b.y);
                            } else {
                                const uint4 b = bm < M ? lds128(b_base + ks * 64) : make_uint4(0u, 0u, 0u, 0u);
                                mma_bf16(accs[0], a, b.x, b.y);
                                mma_bf16(accs[1], a, b.z, b.w);
                            }
                        }
                        break;
                    }
                    uint32_t a[4][4];
                    if (packed) {
                        uint2 b[4];
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            ldmatrix_x4(a_base + ks * 32, a[ks][0], a[ks][1], a[ks][2], a[ks][3]);
                            b[ks] = bm < M ? lds64(b_base + ks * 64) : make_uint2(0u, 0u);
                        }
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) mma_bf16(accs[ks], a[ks], b[ks].x, b[ks].y);
                    } else {
                        uint4 b[4];
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            ldmatrix_x4(a_base + ks * 32, a[ks][0], a[ks][1], a[ks][2], a[ks][3]);
                            b[ks] = bm < M ? lds128(b_base + ks * 64) : make_uint4(0u, 0u, 0u, 0u);
                        }
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            mma_bf16(accs[(ks & 1) * 2], a[ks], b[ks].x, b[ks].y);
                            mma_bf16(accs[(ks & 1) * 2 + 1], a[ks], b[ks].z, b[ks].w);
                        }
                    }
                    a_base += 4 * 32;
                    b_base += 4 * 64;
                }
            }
            // the stage goes back to the producer as soon as this warp has read its slice
            __syncwarp();
            if (lane == 0) mbar_arrive(&c->empty[pos.stage]);
            pos.advance();
        }
        // ---- hand the partial tile to the finisher.  Four slots round-robin; a slot is reused
        // four groups later, once the finisher has freed it (it almost always has). ----
        const int sl = g & 3;
        const int lost = DIRECT ? *(volatile int*)&c->flag : 0;
        ok = wait_barrier(p, c, &c->slot_free[sl], ((pos.comb >> sl) & 1u) ^ 1u, seq, WHERE_COMBINE) && ok;
        if (DIRECT && lost < 0) return;                                      // values of x never came (set before the barrier above): nothing is stored
        pos.comb ^= 1u << sl;
        sts_volatile4(&red[sl * (8 * 32) + warp * 32 + lane],
                      make_float4((accs[0][0] + accs[1][0]) + (accs[2][0] + accs[3][0]), (accs[0][1] + accs[1][1]) + (accs[2][1] + accs[3][1]),
                                  (accs[0][2] + accs[1][2]) + (accs[2][2] + accs[3][2]), (accs[0][3] + accs[1][3]) + (accs[2][3] + accs[3][3])));
        __syncwarp();
        if (lane == 0) mbar_arrive(&c->slot_full[sl]);                        // release: the warp's deposit
    }
    // the instruction's results are in memory when the finisher says so
    wait_barrier(p, c, &c->epi_done, (pos.comb >> 4) & 1u, seq, WHERE_COMBINE);
    pos.comb ^= 16u;
    phase_mark(p, c, 2);
}

// an instruction's whole wait list, by the calling warp
static __device__ __noinline__ bool wait_list(const Params& p, Ctrl* c, int nwait, int wait_off, int seq) {
    bool ok = true;
    for (int k = threadIdx.x & 31; k < nwait; k += 32) {
        const int2 w = __ldg(p.waits + wait_off + k);
        ok = wait_counter(p, c, w.x, w.y, seq) && ok;
    }
    return __all_sync(0xffffffffu, ok) != 0;
}

// The finisher warp: walks the CTA's instructions like the producer does and, for every streaming
// linear of the tensor-core path, turns the deposited partial tiles into outputs.
// Lane l holds rows ob = o0 + 16 * group + (l >> 2) and ob + 8, activation rows m0 = 2 * (l & 3), m0 + 1
// (the MMA result layout); with packed activations (M <= 4) lanes l & 3 >= 2 hold low-part products.
__device__ __forceinline__ void gemv_finisher(const Params& p, Ctrl* c, uint8_t* work) {
    const int lane = threadIdx.x & 31;
    const float4* red = reinterpret_cast<const float4*>(work + kMmaRedOff);
    const float* rowstat = reinterpret_cast<const float*>(work + kMmaStatOff);
    uint32_t fullpar = 0;                                                     // parities of slot_full[0..3], bit 4: deps_met
    for (int idx = blockIdx.x; idx < p.n_insts; idx += gridDim.x) {
        const Inst in = fetch_inst(p, idx);
        const int opi = in.opi - 1;
        if (opi < 0 || opi >= p.n_ops) return;
        const mk_op_desc* op = p.ops + opi;
        if (op->kind != MK_OP_GEMV || !(op->flags & GEMV_F_UNITS)) continue;
        const int M = op->i[0], K = op->i[2], act = op->i[3], odt = op->i[5], rdt = op->i[6];
        const bool swi = op->flags & GEMV_F_SWIGLU, rms = op->flags & GEMV_F_RMS;
        const int o0 = in.a0, o1 = in.a1, seq = in.seq;
        const int ngroups = (swi ? 2 : 1) * ((o1 - o0 + 15) / 16);
        const void* biasp = reinterpret_cast<const void*>(op->ptr[3]);
        const bool direct_out = op->flags & GEMV_F_DIRECT_OUT, direct_res = op->flags & GEMV_F_DIRECT_RES;
        const void* resp = reinterpret_cast<const void*>(op->ptr[4] + (direct_res ? p.direct_off : 0));
        void* outp = reinterpret_cast<void*>(op->ptr[2] + (direct_out ? p.direct_off : 0));
        const long long ldo = op->ld[2], ldr = op->ld[4];
        const float eps = op->f[0];
        const bool packed = M <= 4;
        const int m0 = 2 * (lane & 3);
        const bool storer = !(packed && (lane & 3) >= 2);
        float rs[2] = {1.f, 1.f};
        float gate[4] = {0.f, 0.f, 0.f, 0.f};
        // this lane's arrival target, read now so that it is in a register when the last store has left
        const int arrive_to = lane < in.narrive ? __ldg(p.arrives + in.arrive_off + lane) : -1;
        // Operands of the epilogue may be results of earlier instructions: nothing is read before
        // the compute warps have seen the instruction's dependencies met.
        bool ok = wait_barrier(p, c, &c->deps_met, (fullpar >> 4) & 1u, seq, WHERE_COMBINE, 2);
        fullpar ^= 16u;
        if (!ok) return;
        // (the compute warps look at a direct x alone)
        if ((op->flags & GEMV_F_DIRECT_X) && in.nwait > 0 && !wait_list(p, c, in.nwait, in.wait_off, seq)) return;
        // (a direct residual was written hops ago: not there only when a program's first ops are late)
        auto residual = [&](long long e) {
            if (!direct_res) return load1(resp, e, rdt);
            const float* at = reinterpret_cast<const float*>(resp) + e;
            float v = load1_direct(at);
            if (__float_as_uint(v) == kUnwritten) {
                v = wait1_direct(p, c, at, seq);
                if (__float_as_uint(v) == kUnwritten) ok = false;
            }
            return v;
        };
#pragma unroll 1
        for (int g = 0; g < ngroups; ++g) {
            const int sl = g & 3;
            const int ob = o0 + (swi ? g >> 1 : g) * 16 + (lane >> 2);
            // epilogue operands are requested before the hand-over wait so their latency is hidden
            float bias_v[2] = {0.f, 0.f}, res_v[4] = {0.f, 0.f, 0.f, 0.f};
            auto fetch_operands = [&]() {
                if (swi || !storer) return;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int o = ob + h * 8;
                    if (o < o1) {
                        if (biasp) bias_v[h] = load1(biasp, o, 0);
                        if (resp) {
                            if (m0 < M) res_v[h * 2] = residual((long long)m0 * ldr + o);
                            if (m0 + 1 < M) res_v[h * 2 + 1] = residual((long long)(m0 + 1) * ldr + o);
                        }
                    }
                }
            };
            fetch_operands();
            ok = wait_barrier(p, c, &c->slot_full[sl], (fullpar >> sl) & 1u, seq, WHERE_COMBINE, 2) && ok;
            fullpar ^= 1u << sl;
            if (!__all_sync(0xffffffffu, ok)) return;                         // the launch is failing (no lane stays behind, or stores the marker)
            if (g == 0) {
                if (rms && storer) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (m0 + j < M) {
                            float sq = 0.f;
#pragma unroll
                            for (int w8 = 0; w8 < kComputeWarps; ++w8) sq += rowstat[w8 * 8 + m0 + j];
                            rs[j] = rsqrt_approx(sq / (float)K + eps);
                        }
                    }
                }
            }
            float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int w8 = 0; w8 < kComputeWarps; ++w8) {
                const float4 q = lds_volatile4(&red[sl * (8 * 32) + w8 * 32 + lane]);
                v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&c->slot_free[sl]);                    // the slot has been read
            if (packed) {
                // columns 4..7 hold the low-part products of rows 0..3: add them to columns 0..3,
                // which sit two lanes further down in the quad
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] += __shfl_xor_sync(0xffffffffu, v[e], 2);
            }
            if (storer) {
                // v[0], v[1]: row ob, activation rows m0, m0 + 1;  v[2], v[3]: row ob + 8
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int o = ob + (e >> 1) * 8, m = m0 + (e & 1);
                    const float y = v[e] * rs[e & 1];
                    if (swi && !(g & 1)) {
                        gate[e] = y;
                    } else if (o < o1 && m < M) {
                        const float r = swi ? gate[e] * sigmoidf_(gate[e]) * y : apply_act(act, y + bias_v[e >> 1]) + res_v[e];
                        if (direct_out) store1_direct(reinterpret_cast<float*>(outp) + (long long)m * ldo + o, r);
                        else store1(outp, (long long)m * ldo + o, odt, r);
                    }
                }
            }
        }
        // The instruction's arrivals leave from here, right behind its last store: __syncwarp orders
        // every lane's stores before the arriving lanes' red.release.gpu, whose release is cumulative
        // over them.  (More than 32 targets: the compute warps send the rest, see the wrapper.)
        __syncwarp();
        if (lane == 0) mbar_arrive(&c->epi_done);                             // shared memory is free: the compute warps move on
        if (arrive_to >= 0) red_release_add(p.counters + arrive_to, 1);
    }
}

}  // namespace mk
