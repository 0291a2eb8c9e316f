// Norms over many rows and pointwise tiles: ops that stream activations through an SM (MK_OP_NORM with eight or more rows
// per instruction, MK_OP_ELTWISE).  At the sizes of a prefill or DiT block they are bound by L2 / HBM bandwidth only if an
// instruction keeps enough of it in flight: an instruction of 8 rows x 1024 columns (one row per warp) took 7.5 us, of
// 32 x 512 gated elements 9.6 us, nearly all of it one L2 round trip behind the other plus what an instruction costs
// whatever its size.  So the schedule gives each SM about one instruction per op (schedule.py norm_rows, ew_rows), a warp
// requests several rows before it uses the first, operands that all rows share are loaded once per instruction, and the
// bodies keep the CTA's walk for as long as the next instruction is of the same kind (walk.cuh).
#pragma once
#include <type_traits>
#include "mk_device.cuh"
#include "ops.cuh"

namespace mk {

// (Loads are unconditional, with the row or column clamped to the last one: under the condition of their use the compiler
// moves them there, one round trip behind the other.)
constexpr int kEwCols = 512;                               // config.py EW_COLS
enum { EW_UNARY = 0, EW_BINARY, EW_SWIGLU, EW_MODULATE, EW_ROPE, EW_GATED };
enum { BIN_ADD = 0, BIN_SUB, BIN_MUL, BIN_MAX, BIN_MIN };

__device__ __forceinline__ float apply_bin(int fn, float a, float b) {
    switch (fn) {
        case BIN_ADD: return a + b;
        case BIN_SUB: return a - b;
        case BIN_MUL: return a * b;
        case BIN_MAX: return fmaxf(a, b);
        default: return fminf(a, b);
    }
}

// Binary / modulate tile whose rows all read ONE row of the second (and third) operand -- a per-image gate, scale or
// shift over that image's tokens: the thread keeps its 8 columns of them and streams a, eight rows in flight when a is 16-bit.
template <int MODE>
__device__ __forceinline__ void eltwise_tile_one_group(const mk_op_desc* op, int r0, int col, int rows, int rowp, int rpp) {
    const int fn = op->i[3], group = op->i[4];
    const int adt = op->i[6], bdt = op->i[7], cdt = op->i[8], odt = op->i[9];
    const void* A = reinterpret_cast<const void*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[3]);
    const long long grow = r0 / group;
    float b[8], cc[8];
    load8(reinterpret_cast<const void*>(op->ptr[1]), grow * op->ld[1] + col, bdt, b);
    if (MODE == EW_MODULATE) {
        load8(reinterpret_cast<const void*>(op->ptr[2]), grow * op->ld[2] + col, cdt, cc);
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] += 1.0f;
    }
    auto body = [&](auto tag) {
        constexpr bool S16 = decltype(tag)::value;
        constexpr int UN = S16 ? 8 : 4;
        for (int rr = rowp; rr < rows; rr += UN * rpp) {
            Raw8x<S16> ra[UN];
#pragma unroll
            for (int u = 0; u < UN; ++u) ra[u].load(A, (long long)(r0 + min(rr + u * rpp, rows - 1)) * op->ld[0] + col, adt);
#pragma unroll
            for (int u = 0; u < UN; ++u) {
                if (rr + u * rpp >= rows) continue;
                float a[8];
                ra[u].unpack(adt, a);
                if (MODE == EW_MODULATE) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] = fmaf(a[e], b[e], cc[e]);
                } else if (fn == BIN_MUL) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] *= b[e];
                } else if (fn == BIN_ADD) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] += b[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) a[e] = apply_bin(fn, a[e], b[e]);
                }
                store8(O, (long long)(r0 + rr + u * rpp) * op->ld[3] + col, odt, a);
            }
        }
    };
    if (adt != DT_F32) body(std::true_type{});
    else body(std::false_type{});
}

// One tile of a pointwise op other than rope.  A pointwise instruction is a few thousand elements; with the mode, the
// function and the tile geometry as run-time switches and divisions inside the vector loop it was instruction-bound
// (8.7 us for a 32 x 512 modulate tile: ~300 instructions per 8-element vector at a fraction of an instruction per
// cycle).  Here the mode is a template parameter, the function is switched once
// per vector, a thread keeps its columns and walks rows (no division in the loop), and two rows are in flight.
template <int MODE, bool SIXTEEN>
__device__ __forceinline__ void eltwise_tile(const mk_op_desc* op, int r0, int c0, int rows, int cols) {
    const int fn = op->i[3], group = op->i[4];
    const int adt = op->i[6], bdt = op->i[7], cdt = op->i[8], odt = op->i[9];
    const void* A = reinterpret_cast<const void*>(op->ptr[0]);
    const void* B = reinterpret_cast<const void*>(op->ptr[1]);
    const void* Cp = reinterpret_cast<const void*>(op->ptr[2]);
    void* O = reinterpret_cast<void*>(op->ptr[3]);
    constexpr bool HASB = MODE != EW_UNARY, HASC = MODE == EW_MODULATE, GROUPED = MODE == EW_BINARY || MODE == EW_MODULATE;
    const int vpr = cols >> 3;                                   // vectors per row: at most 64
    // threads cover whole rows side by side: thread -> (row of the pass, vector of the row)
    const int tpr = vpr <= 1 ? 1 : vpr <= 2 ? 2 : vpr <= 4 ? 4 : vpr <= 8 ? 8 : vpr <= 16 ? 16 : vpr <= 32 ? 32 : 64;   // threads per row
    const int rpp = kComputeThreads / tpr;                       // rows per pass
    const int vec = threadIdx.x & (tpr - 1), rowp = threadIdx.x / tpr;
    if (vec >= vpr) return;
    const int col = c0 + vec * 8;
    if (GROUPED && (r0 / group) == ((r0 + rows - 1) / group)) {
        // every row of the tile reads the same row of b (and c): a thread's column of them is loaded once, and only a streams
        eltwise_tile_one_group<MODE>(op, r0, col, rows, rowp, rpp);
        return;
    }
    // rows in flight per thread: with 16-bit operands a vector is four registers and a thread's whole share of the tile
    // (eight rows) fits; otherwise two (more spill, and a spill is an L2 round trip like the loads it was to hide)
    constexpr int UN = SIXTEEN ? (HASC ? 2 : HASB ? 4 : 8) : 2;
    for (int rr = rowp; rr < rows; rr += UN * rpp) {
        Raw8x<SIXTEEN> ra[UN], rb[HASB ? UN : 1], rc[HASC ? UN : 1];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int r = r0 + min(rr + u * rpp, rows - 1);
            ra[u].load(A, (long long)r * op->ld[0] + col, adt);
            const long long rb_row = GROUPED ? r / group : r;
            if (HASB) rb[u].load(B, rb_row * op->ld[1] + col, bdt);
            if (HASC) rc[u].load(Cp, rb_row * op->ld[2] + col, cdt);
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int r = r0 + rr + u * rpp;
            if (rr + u * rpp >= rows) continue;
            float a[8], b[8], cc[8];
            ra[u].unpack(adt, a);
            if (HASB) rb[u].unpack(bdt, b);
            if (MODE == EW_UNARY) {
                switch (fn) {
                    case ACT_NONE: break;
                    case ACT_SILU:
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] = a[e] * sigmoidf_(a[e]);
                        break;
                    default:
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] = apply_act(fn, a[e]);
                }
            } else if (MODE == EW_BINARY) {
                switch (fn) {
                    case BIN_ADD:
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] += b[e];
                        break;
                    case BIN_MUL:
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] *= b[e];
                        break;
                    default:
#pragma unroll
                        for (int e = 0; e < 8; ++e) a[e] = apply_bin(fn, a[e], b[e]);
                }
            } else if (MODE == EW_SWIGLU) {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = apply_act(fn, a[e]) * b[e];
            } else {  // EW_MODULATE: x * (1 + scale[g]) + shift[g]
                rc[u].unpack(cdt, cc);
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = fmaf(a[e], 1.0f + b[e], cc[e]);
            }
            store8(O, (long long)r * op->ld[3] + col, odt, a);
        }
    }
}

// EW_GATED: out = fn(a, b * c[r / group]) -- a gated residual, x + y * gate[image] (passes.fuse_pointwise).  a and b
// stream, the gate row of a tile is loaded once when the tile lies in one group.
template <bool SIXTEEN>
__device__ __forceinline__ void eltwise_tile_gated(const mk_op_desc* op, int r0, int c0, int rows, int cols) {
    const int fn = op->i[3], group = op->i[4];
    const int adt = op->i[6], bdt = op->i[7], cdt = op->i[8], odt = op->i[9];
    const void* A = reinterpret_cast<const void*>(op->ptr[0]);
    const void* B = reinterpret_cast<const void*>(op->ptr[1]);
    const void* G = reinterpret_cast<const void*>(op->ptr[2]);
    void* O = reinterpret_cast<void*>(op->ptr[3]);
    const int vpr = cols >> 3;
    const int tpr = vpr <= 1 ? 1 : vpr <= 2 ? 2 : vpr <= 4 ? 4 : vpr <= 8 ? 8 : vpr <= 16 ? 16 : vpr <= 32 ? 32 : 64;
    const int rpp = kComputeThreads / tpr;
    const int vec = threadIdx.x & (tpr - 1), rowp = threadIdx.x / tpr;
    if (vec >= vpr) return;
    const int col = c0 + vec * 8;
    const bool one = (r0 / group) == ((r0 + rows - 1) / group);
    float gt[8];
    if (one) load8(G, (long long)(r0 / group) * op->ld[2] + col, cdt, gt);
    constexpr int UN = SIXTEEN ? 6 : 2;
    for (int rr = rowp; rr < rows; rr += UN * rpp) {
        Raw8x<SIXTEEN> ra[UN], rb[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int r = r0 + min(rr + u * rpp, rows - 1);
            ra[u].load(A, (long long)r * op->ld[0] + col, adt);
            rb[u].load(B, (long long)r * op->ld[1] + col, bdt);
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int r = r0 + rr + u * rpp;
            if (rr + u * rpp >= rows) continue;
            float a[8], b[8];
            ra[u].unpack(adt, a);
            rb[u].unpack(bdt, b);
            if (!one) load8(G, (long long)(r / group) * op->ld[2] + col, cdt, gt);
            if (fn == BIN_ADD) {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = fmaf(b[e], gt[e], a[e]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = apply_bin(fn, a[e], b[e] * gt[e]);
            }
            store8(O, (long long)r * op->ld[3] + col, odt, a);
        }
    }
}

// A vector of 8 elements of a type known at compile time.  The bodies below are a loop over rows of a few hundred instructions:
// with the element types as run-time switches inside an unrolled batch of rows the code was ten times as long, and fetching
// it, not memory, was what an instruction waited for (56 rows of 1024: 30 us, whatever was in flight).
template <int DT> struct Vec8 {
    uint4 v;
    __device__ __forceinline__ void load(const void* base, long long elem) { v = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + elem)); }
    __device__ __forceinline__ void raw(const uint4& w, const uint4&) { v = w; }
    __device__ __forceinline__ void get(float* f) const {
        if (DT == DT_F16) {
            const float2 a = unpack2h(v.x), b = unpack2h(v.y), c = unpack2h(v.z), d = unpack2h(v.w);
            f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
        } else {
            unpack8(v, f);
        }
    }
};
template <> struct Vec8<DT_F32> {
    float4 a, b;
    __device__ __forceinline__ void load(const void* base, long long elem) {
        const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + elem);
        a = __ldcg(p); b = __ldcg(p + 1);
    }
    __device__ __forceinline__ void raw(const uint4& p, const uint4& q) {
        a = make_float4(__uint_as_float(p.x), __uint_as_float(p.y), __uint_as_float(p.z), __uint_as_float(p.w));
        b = make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), __uint_as_float(q.w));
    }
    __device__ __forceinline__ void get(float* f) const { f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w; }
};
template <int DT>
__device__ __forceinline__ void put8(void* base, long long elem, const float* f) {
    uint16_t* p = reinterpret_cast<uint16_t*>(base) + elem;
    *reinterpret_cast<uint4*>(p) = DT == DT_F16 ? make_uint4(pack2h(f[0], f[1]), pack2h(f[2], f[3]), pack2h(f[4], f[5]), pack2h(f[6], f[7])) : pack8(f);
}

// EW_ROPE: rotate-half on whole heads.  A thread keeps its row and its 8 + 8 elements of a head (and the cos / sin values of
// both halves, the same for every head) and walks the tile's heads, the next one requested before this one is used.
template <int XDT, int ODT>
__device__ __forceinline__ void eltwise_tile_rope(const mk_op_desc* op, int r0, int c0, int rows, int cols) {
    const int seq = op->i[4], D = op->i[5], half = D >> 1, hv = half >> 3;           // vectors per half head
    const void* A = reinterpret_cast<const void*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[3]);
    const int heads = cols / D;
    int parts = 1;                                          // threads that share a row's element pair, each with its heads
    while (parts < heads && rows * hv * parts * 2 <= kComputeThreads) parts *= 2;
    const int per = (heads + parts - 1) / parts;
#pragma unroll 1
    for (int u = threadIdx.x; u < rows * hv * parts; u += kComputeThreads) {
        const int r = r0 + u / (hv * parts), rem = u % (hv * parts);
        const int dc = (rem % hv) * 8, h0 = (rem / hv) * per, h1 = min(heads, h0 + per);
        const int tok = r % seq;
        float c1[8], c2[8], s1[8], s2[8];
        const long long row_a = (long long)r * op->ld[0] + c0 + dc, row_o = (long long)r * op->ld[3] + c0 + dc;
        Vec8<XDT> n1, n2;
        if (h0 < h1) {
            n1.load(A, row_a + h0 * D);
            n2.load(A, row_a + h0 * D + half);
        }
        load8(reinterpret_cast<const void*>(op->ptr[1]), (long long)tok * op->ld[1] + dc, op->i[7], c1);
        load8(reinterpret_cast<const void*>(op->ptr[1]), (long long)tok * op->ld[1] + dc + half, op->i[7], c2);
        load8(reinterpret_cast<const void*>(op->ptr[2]), (long long)tok * op->ld[2] + dc, op->i[8], s1);
        load8(reinterpret_cast<const void*>(op->ptr[2]), (long long)tok * op->ld[2] + dc + half, op->i[8], s2);
#pragma unroll 1
        for (int h = h0; h < h1; ++h) {
            float x1[8], x2[8], o[8];
            n1.get(x1);
            n2.get(x2);
            if (h + 1 < h1) {
                n1.load(A, row_a + (h + 1) * D);
                n2.load(A, row_a + (h + 1) * D + half);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = x1[e] * c1[e] - x2[e] * s1[e];
            store8(O, row_o + h * D, ODT, o);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = x2[e] * c2[e] + x1[e] * s2[e];
            store8(O, row_o + h * D + half, ODT, o);
        }
    }
}

// MK_OP_ELTWISE.  ptr 0 a (x / gate), 1 b (b / up / scale / cos), 2 c (shift / sin), 3 out
// i 0 R, 1 C, 2 mode, 3 fn (activation or binary code), 4 group (rows of a per row of b; rope: seq),
//   5 head_dim (rope), 6..9 dtypes of a, b, c, out (DT_*), 10 rows per instruction.  args: 0 row tile, 1 col tile.
// Variant: mode | 16 when every operand the tile streams is 16-bit; rope: mode | x dtype << 4 | out dtype << 6.  (A function, and a
// register allocation, per variant: op_stream.cu.)
__device__ __forceinline__ int ew_variant(const mk_op_desc* op) {
    const int mode = op->i[2], adt = op->i[6], bdt = op->i[7], cdt = op->i[8];
    if (mode == EW_ROPE) return mode | adt << 4 | op->i[9] << 6;
    const bool all16 = adt != DT_F32 && (mode == EW_UNARY || bdt != DT_F32) && (mode != EW_MODULATE || cdt != DT_F32);
    return mode | (all16 ? 16 : 0);
}
template <int V>
__device__ __forceinline__ void op_eltwise(const mk_op_desc* op, int a0, int a1) {
    constexpr int mode = V & 15;
    const int R = op->i[0], Cc = op->i[1], tr = op->i[10];
    const int r0 = a0 * tr, c0 = a1 * kEwCols;
    const int rows = min(tr, R - r0), cols = min(kEwCols, Cc - c0);
    if constexpr (mode == EW_ROPE) eltwise_tile_rope<((V >> 4) & 3), ((V >> 6) & 3)>(op, r0, c0, rows, cols);
    else if constexpr (mode == EW_GATED) eltwise_tile_gated<(V & 16) != 0>(op, r0, c0, rows, cols);
    else eltwise_tile<mode, (V & 16) != 0>(op, r0, c0, rows, cols);
}

// ---- norms ---------------------------------------------------------------------------------------------------------------------
// MK_OP_NORM with i 3 >= 8 rows per instruction (descriptor: op_pointwise.cuh): rows r0 + warp, + 8, ..., a row per warp.  Bound by
// memory latency: an SM gets what it has requested per round trip (2 us with all SMs streaming), so each warp keeps 12 KB of
// rows on their way through the work area (DEEP; 64 rows of 2048 fp16: 26.8 -> 14.4 us).  A lane reads back what it
// copied itself.  With one or two rows per warp there is nothing to run ahead of: the next row in registers (8 rows 5.1 us, 6.0
// through the work area).  Gain, and scale and shift of the current
// group of rows, stay in registers.  NPER: 8-element vectors of a row per lane.  HW: gain.  MOD: scale and shift.
constexpr int kNormAhead = 12288;                          // bytes of rows a warp has requested
template <int NPER, int XDT, int ODT, bool HW, bool MOD, bool DEEP>
__device__ __forceinline__ void norm_stream(const mk_op_desc* op, int r0, int rows) {
    constexpr bool kAhead = !DEEP && (XDT != DT_F32 || NPER <= 4);    // (two fp32 rows of 2048 do not fit)
    constexpr int kPlanes = XDT == DT_F32 ? 2 : 1, kRow = NPER * kPlanes * 512, kDepth = kNormAhead / kRow;     // 16 bytes of a vector per plane
    static_assert(kDepth >= 1 && kTcXOff + kComputeWarps * kNormAhead <= kWorkBytes, "norm rows exceed the work area");
    const int Cc = op->i[1], rms = op->i[2], group = max(1, op->i[6]);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = Cc >> 3;
    const void* X = reinterpret_cast<const void*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[1]);
    const float inv = 1.0f / (float)Cc, eps = op->f[0];
    const long long ldx = op->ld[0], ldo = op->ld[1];
    Vec8<DT_BF16> gw[HW ? NPER : 1];
    float sc[MOD ? NPER * 8 : 1], sh[MOD ? NPER * 8 : 1];
    // (columns beyond the row are clamped to its last vector and left out of the sums and stores)
    auto column = [&](int u) { return (long long)min(lane + u * 32, nvec - 1) * 8; };
    uint8_t* buf = smem_map().work + kTcXOff + warp * kNormAhead + lane * 16;
    Vec8<XDT> x[NPER], nx[kAhead ? NPER : 1];
    auto fetch = [&](int rr, Vec8<XDT>* x) {
#pragma unroll
        for (int u = 0; u < NPER; ++u) x[u].load(X, (r0 + rr) * ldx + column(u));
    };
    auto request = [&](int rr, int slot) {
        if (rr < rows) {
#pragma unroll
            for (int u = 0; u < NPER; ++u)
#pragma unroll
                for (int k = 0; k < kPlanes; ++k)
                    cp_async16(buf + slot * kRow + (u * kPlanes + k) * 512,
                               reinterpret_cast<const uint8_t*>(X) + ((r0 + rr) * ldx + column(u)) * (kPlanes * 2) + k * 16, true);
        }
        cp_async_commit();
    };
    auto modulation = [&](long long g) {
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            load8(reinterpret_cast<const void*>(op->ptr[4]), g * op->ld[4] + column(u), op->i[7], sc + (MOD ? u * 8 : 0));
            load8(reinterpret_cast<const void*>(op->ptr[5]), g * op->ld[5] + column(u), op->i[8], sh + (MOD ? u * 8 : 0));
        }
    };
    if (warp >= rows) return;
    if (DEEP) {
#pragma unroll
        for (int d = 0; d < kDepth; ++d) request(warp + d * kComputeWarps, d);
    } else if (kAhead) {
        fetch(warp, nx);
    }
    int grp = (r0 + warp) / group;
    if (HW) {
#pragma unroll
        for (int u = 0; u < NPER; ++u) gw[HW ? u : 0].load(reinterpret_cast<const void*>(op->ptr[2]), column(u));
    }
    if (MOD) modulation(grp);
    int slot = 0;
#pragma unroll 1
    for (int rr = warp; rr < rows; rr += kComputeWarps) {
        if (DEEP) {
            cp_async_wait<kDepth - 1>();
#pragma unroll
            for (int u = 0; u < NPER; ++u) {
                const uint4* at = reinterpret_cast<const uint4*>(buf + slot * kRow + u * kPlanes * 512);
                x[u].raw(at[0], at[kPlanes == 2 ? 32 : 0]);
            }
            request(rr + kDepth * kComputeWarps, slot);
            if (++slot == kDepth) slot = 0;
        } else if (kAhead) {
#pragma unroll
            for (int u = 0; u < NPER; ++u) x[u] = nx[kAhead ? u : 0];
            fetch(min(rr + kComputeWarps, rows - 1), nx);
        } else {
            fetch(rr, x);
        }
        if (MOD && (r0 + rr) / group != grp) { grp = (r0 + rr) / group; modulation(grp); }
        float s = 0.f, ss = 0.f;
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            float f[8];
            x[u].get(f);
            float a = 0.f, q = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) { a += f[e]; q = fmaf(f[e], f[e], q); }
            const bool in = lane + u * 32 < nvec;
            s += in ? a : 0.f;
            ss += in ? q : 0.f;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        const float mean = rms ? 0.f : s * inv;
        const float rstd = rsqrt_approx(ss * inv - mean * mean + eps);
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            float f[8];
            x[u].get(f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean) * rstd;
            if (HW) {
                float g[8];
                gw[HW ? u : 0].get(g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] *= g[e];
            }
            if (MOD) {
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = fmaf(f[e], 1.0f + sc[MOD ? u * 8 + e : 0], sh[MOD ? u * 8 + e : 0]);
            }
            if (lane + u * 32 < nvec) put8<ODT>(O, (r0 + rr) * ldo + (lane + u * 32) * 8, f);
        }
    }
}

// Any other row (longer than 2048 elements, with a bias, gain and modulation at once, fp32 modulation): two passes over global
// memory, two vectors requested at a time.
__device__ __forceinline__ void norm_two_pass(const mk_op_desc* op, int r0, int rows) {
    const int Cc = op->i[1], rms = op->i[2], xdt = op->i[4], odt = op->i[5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = Cc >> 3;
    const void* X = reinterpret_cast<const void*>(op->ptr[0]);
    const void* W = reinterpret_cast<const void*>(op->ptr[2]);
    const void* Bv = reinterpret_cast<const void*>(op->ptr[3]);
    for (int rr = warp; rr < rows; rr += kComputeWarps) {
        const long long r = r0 + rr, grow = r / max(1, op->i[6]);
        float s = 0.f, ss = 0.f;
        for (int v0 = lane; v0 < nvec; v0 += 64) {
            Raw8 x[2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (v0 + u * 32 < nvec) x[u] = load8_raw(X, r * op->ld[0] + (v0 + u * 32) * 8, xdt);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (v0 + u * 32 >= nvec) continue;
                float f[8];
                unpack8_raw(x[u], xdt, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) { s += f[e]; ss += f[e] * f[e]; }
            }
        }
        s = warp_sum(s);
        ss = warp_sum(ss);
        const float mean = rms ? 0.f : s / (float)Cc;
        const float rstd = rsqrt_approx(ss / (float)Cc - mean * mean + op->f[0]);
        for (int v = lane; v < nvec; v += 32) {
            float f[8], g[8], h[8];
            load8(X, r * op->ld[0] + v * 8, xdt, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean) * rstd;
            if (W) {
                load8(W, v * 8, DT_BF16, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] *= g[e];
            }
            if (Bv) {
                load8(Bv, v * 8, DT_BF16, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += g[e];
            }
            if (op->ptr[4]) {
                load8(reinterpret_cast<const void*>(op->ptr[4]), grow * op->ld[4] + v * 8, op->i[7], g);
                load8(reinterpret_cast<const void*>(op->ptr[5]), grow * op->ld[5] + v * 8, op->i[8], h);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = fmaf(f[e], 1.0f + g[e], h[e]);
            }
            store8(reinterpret_cast<void*>(op->ptr[1]), r * op->ld[1] + v * 8, odt, f);
        }
    }
}

// Variant of a norm: x dtype (bits 0-1), fp16 output (bit 2), vectors per lane (bit 3: 8, else 4), gain (bit 4), modulation (bit 5),
// three or more rows per warp (bit 6)
constexpr int NORM_DEEP = 64, NORM_ANY = 128;
__device__ __forceinline__ int norm_variant(const mk_op_desc* op) {
    const int nper = ((op->i[1] >> 3) + 31) / 32;
    const bool w = op->ptr[2] != 0, mod = op->ptr[4] != 0;
    if (op->ptr[3] || (w && mod) || op->i[5] == DT_F32 || nper > (mod ? 4 : 8)) return NORM_ANY;
    return (op->i[3] > 2 * kComputeWarps ? NORM_DEEP : 0) | op->i[4] | (op->i[5] == DT_F16 ? 4 : 0) | (nper > 4 ? 8 : 0) | (w ? 16 : 0) | (mod ? 32 : 0);
}
template <int V>
__device__ __forceinline__ void op_norm_rows(const mk_op_desc* op, int a0) {
    const int r0 = a0 * op->i[3], rows = min(op->i[3], op->i[0] - r0);
    if constexpr (V == NORM_ANY) norm_two_pass(op, r0, rows);
    else norm_stream<(V & 8) ? 8 : 4, V & 3, (V & 4) ? DT_F16 : DT_BF16, (V & 16) != 0, (V & 32) != 0, (V & NORM_DEEP) != 0>(op, r0, rows);
}

}  // namespace mk
