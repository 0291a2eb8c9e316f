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
// memory latency: an SM gets what it has requested per round trip (2 us with all SMs streaming), so each warp keeps 10 to 12 KB of
// rows on their way through the work area (64 rows of 2048 fp16 one row ahead: 26.8 us, so 14.4).  A lane reads back what it copied
// itself, twice: for the sums and for the result.
// The body runs once per op on an SM, between bodies with other registers, so what it keeps in registers is saved and restored around it
// and what it unrolls is fetched cold: with a row, the gain and the group's scale and shift in registers it saved 296 to 464 bytes per
// thread and took 7 us to its first row (64 rows of 1024, DiT).  So the gain, or scale and shift of the rows' group, are in shared memory
// too: 8 bytes saved, the op 20 -> 15 us (with what lies between it and the linear in front of it), DiT of 32 images 8409 -> 8164, of 4 images
// 3453 -> 3158, MLP block of 3001 rows 197.5 -> 193.5 us.
// NPER: 8-element vectors of a row per lane.  HW: gain.  MOD: scale and shift.
template <int NPER, int XDT, int ODT, bool HW, bool MOD>
__device__ __forceinline__ void norm_stream(const mk_op_desc* op, int r0, int rows) {
    constexpr int kShared = MOD ? NPER * 2048 : HW ? NPER * 512 : 0;         // bytes of gain, or of scale and shift as fp32
    constexpr int kAhead = (kWorkBytes - kTcXOff - kShared) / kComputeWarps;  // ... of rows a warp has requested
    constexpr int kPlanes = XDT == DT_F32 ? 2 : 1, kRow = NPER * kPlanes * 512, kDepth = kAhead / kRow;      // 16 bytes of a vector per plane
    constexpr int kSharedOff = kTcXOff + kComputeWarps * kDepth * kRow;
    static_assert(kDepth >= 1 && kSharedOff + kShared <= kWorkBytes, "norm rows exceed the work area");
    const int Cc = op->i[1], rms = op->i[2], group = MOD ? max(1, op->i[6]) : op->i[0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = Cc >> 3;
    const float inv = 1.0f / (float)Cc, eps = op->f[0];
    const long long ldx = op->ld[0], ldo = op->ld[1];
    // (columns beyond the row are clamped to its last vector and left out of the sums and stores)
    auto column = [&](int u) { return min(lane + u * 32, nvec - 1) * 8; };
    uint8_t* work = smem_map().work;
    uint8_t* buf = work + kTcXOff + warp * (kDepth * kRow) + lane * 16;
    uint8_t* shared = work + kSharedOff;                      // (lane's vectors as in the rows; scale and shift: four planes of 16 bytes per vector)
    auto request = [&](int rr, int slot) {
        if (rr < rows) {
            const uint8_t* from = reinterpret_cast<const uint8_t*>(op->ptr[0]) + (r0 + rr) * ldx * (kPlanes * 2);
#pragma unroll
            for (int u = 0; u < NPER; ++u)
#pragma unroll
                for (int k = 0; k < kPlanes; ++k) cp_async16(buf + slot * kRow + (u * kPlanes + k) * 512, from + column(u) * (kPlanes * 2) + k * 16, true);
        }
        cp_async_commit();
    };
    int next = warp, slot = 0, rr = warp;
    // (the gain travels with the first rows, and is waited for between a warp's first sums and its first result)
    bool gain_there = !HW;
    if (HW)
        for (int v = threadIdx.x; v < NPER * 32; v += kComputeThreads)
            cp_async16(shared + v * 16, reinterpret_cast<const uint8_t*>(op->ptr[2]) + min(v, nvec - 1) * 16, true);
#pragma unroll 1
    for (int d = 0; d < kDepth; ++d, next += kComputeWarps) request(next, d);
#pragma unroll 1
    for (int grp = r0 / group;; ++grp) {
        const int end = MOD ? min(rows, (grp + 1) * group - r0) : rows;          // the instruction's rows of this group (most have one group)
        if (MOD) {
            if (grp > r0 / group) compute_sync();                                // (the group before has been read)
            for (int v = threadIdx.x; v < 2 * NPER * 32; v += kComputeThreads) {
                const int which = v >= NPER * 32, u = v - which * NPER * 32;
                float f[8];
                load8(reinterpret_cast<const void*>(op->ptr[4 + which]), (long long)grp * op->ld[4 + which] + min(u, nvec - 1) * 8, op->i[7 + which], f);
                float4* to = reinterpret_cast<float4*>(shared) + which * NPER * 64 + u;
                to[0] = make_float4(f[0], f[1], f[2], f[3]);
                to[NPER * 32] = make_float4(f[4], f[5], f[6], f[7]);
            }
            compute_sync();
        }
#pragma unroll 1
        for (; rr < end; rr += kComputeWarps, next += kComputeWarps) {
            cp_async_wait<kDepth - 1>();
            const uint8_t* at = buf + slot * kRow;
            auto row = [&](int u, float* f) {
                Vec8<XDT> x;
                x.raw(*reinterpret_cast<const uint4*>(at + u * kPlanes * 512), *reinterpret_cast<const uint4*>(at + u * kPlanes * 512 + (kPlanes - 1) * 512));
                x.get(f);
            };
            float s = 0.f, ss = 0.f;
#pragma unroll 4
            for (int u = 0; u < NPER; ++u) {
                float f[8];
                row(u, f);
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
            const long long out = (r0 + rr) * ldo;
            if (!gain_there) {
                compute_sync();
                gain_there = true;
            }
#pragma unroll 2
            for (int u = 0; u < NPER; ++u) {
                float f[8], g[8], h[8];
                row(u, f);
                if (HW) unpack8(reinterpret_cast<const uint4*>(shared)[u * 32 + lane], g);
                if (MOD) {
                    const float4* from = reinterpret_cast<const float4*>(shared) + u * 32 + lane;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float4 q = from[k * NPER * 32], r = from[(2 + k) * NPER * 32];
                        g[4 * k] = q.x; g[4 * k + 1] = q.y; g[4 * k + 2] = q.z; g[4 * k + 3] = q.w;
                        h[4 * k] = r.x; h[4 * k + 1] = r.y; h[4 * k + 2] = r.z; h[4 * k + 3] = r.w;
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    f[e] = (f[e] - mean) * rstd;
                    if (HW) f[e] *= g[e];
                    if (MOD) f[e] = fmaf(f[e], 1.0f + g[e], h[e]);
                }
                if (lane + u * 32 < nvec) put8<ODT>(reinterpret_cast<void*>(op->ptr[1]), out + (lane + u * 32) * 8, f);
            }
            request(next, slot);
            if (++slot == kDepth) slot = 0;
        }
        if (end >= rows) break;
    }
    if (!gain_there) {                                                           // (a warp without a row)
        cp_async_wait<0>();
        compute_sync();
    }
}

// Plain rows, several per warp (with a gain more than four, without more than one): the row stays in registers, so that it is read from shared memory
// once and its place is requested again before the sums; 200 bytes per thread saved around it are little beside as many rows.  us per norm in a chain
// of them, norm_stream / here: 9600 rows of 2048 with a gain 16.9 / 14.0, of 1024 10.4 / 9.1, of 1152 16.5 / 15.0; without one 9600 of 2048
// 14.3 / 12.1, of 1152 14.0 / 13.1, 1200 of 1024 3.8 / 3.6.  (Addresses in 64 bits from the start: in 32 the unmodulated rows of 2048 took 13.1.)  Prompts and MLP blocks the same (4 x 4096 tokens 9209 and 9246 us, runs differ by 1 %).  With a
// gain and up to four rows per warp norm_stream is ahead where other ops lie between (MLP block of 2400 rows 161, 165 in this form).
template <int NPER, int XDT, int ODT, bool HW>
__device__ __forceinline__ void norm_kept_rows(const mk_op_desc* op, int r0, int rows) {
    constexpr int kGain = HW ? NPER * 512 : 0, kPlanes = XDT == DT_F32 ? 2 : 1, kRow = NPER * kPlanes * 512;
    constexpr int kDepth = (kWorkBytes - kTcXOff - kGain) / kComputeWarps / kRow, kGainOff = kTcXOff + kComputeWarps * kDepth * kRow;
    static_assert(kDepth >= 1 && kGainOff + kGain <= kWorkBytes, "norm rows exceed the work area");
    const int Cc = op->i[1], rms = op->i[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = Cc >> 3;
    const float inv = 1.0f / (float)Cc, eps = op->f[0];
    const long long ldx = op->ld[0], ldo = op->ld[1];
    const uint8_t* X = reinterpret_cast<const uint8_t*>(op->ptr[0]);
    void* O = reinterpret_cast<void*>(op->ptr[1]);
    auto column = [&](int u) { return (long long)min(lane + u * 32, nvec - 1) * 8; };
    uint8_t* buf = smem_map().work + kTcXOff + warp * (kDepth * kRow) + lane * 16;
    auto request = [&](int rr, int slot) {
        if (rr < rows) {
#pragma unroll
            for (int u = 0; u < NPER; ++u)
#pragma unroll
                for (int k = 0; k < kPlanes; ++k)
                    cp_async16(buf + slot * kRow + (u * kPlanes + k) * 512, X + ((r0 + rr) * ldx + column(u)) * (kPlanes * 2) + k * 16, true);
        }
        cp_async_commit();
    };
    uint8_t* gain = smem_map().work + kGainOff;
    if (HW)
        for (int v = threadIdx.x; v < NPER * 32; v += kComputeThreads)
            cp_async16(gain + v * 16, reinterpret_cast<const uint8_t*>(op->ptr[2]) + min(v, nvec - 1) * 16, true);
#pragma unroll
    for (int d = 0; d < kDepth; ++d) request(warp + d * kComputeWarps, d);
    if (HW) {
        cp_async_wait<kDepth - 1>();
        compute_sync();
    }
    int slot = 0;
#pragma unroll 1
    for (int rr = warp; rr < rows; rr += kComputeWarps) {
        cp_async_wait<kDepth - 1>();
        Vec8<XDT> x[NPER];
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            const uint4* at = reinterpret_cast<const uint4*>(buf + slot * kRow + u * kPlanes * 512);
            x[u].raw(at[0], at[kPlanes == 2 ? 32 : 0]);
        }
        request(rr + kDepth * kComputeWarps, slot);
        if (++slot == kDepth) slot = 0;
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
                unpack8(reinterpret_cast<const uint4*>(gain)[u * 32 + lane], g);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] *= g[e];
            }
            if (lane + u * 32 < nvec) put8<ODT>(O, (r0 + rr) * ldo + (lane + u * 32) * 8, f);
        }
    }
}

// Modulated rows whose scale and shift rows change with every row or every two or three (up to 1024 columns): each warp requests its row's own in front
// of the sums, into registers.  In shared memory, as above, they change up to eight times in eight rows, with two barriers and a round
// trip to L2 each.  us per norm, above / here: 9600 rows of 1024 with a scale row each 102 / 23, of 512 80 / 20, 1200 rows of 1024 20 / 5.9, 300 rows
// 7.2 / 6.9; two rows per scale row 49 / 21, 42 / 20, 11 / 5.9, 6.9 / 6.9.  (256 bytes per thread are saved around this body; four rows per scale row take
// 7.1 above for 1200 rows of 1024, less than the 7.4 they took with everything in registers.)
template <int XDT, int ODT>
__device__ __forceinline__ void norm_own(const mk_op_desc* op, int r0, int rows) {
    constexpr int NPER = 4, kPlanes = XDT == DT_F32 ? 2 : 1, kRow = NPER * kPlanes * 512, kDepth = (kWorkBytes - kTcXOff) / kComputeWarps / kRow;
    const int Cc = op->i[1], rms = op->i[2], group = max(1, op->i[6]);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = Cc >> 3;
    const float inv = 1.0f / (float)Cc, eps = op->f[0];
    const long long ldx = op->ld[0], ldo = op->ld[1];
    auto column = [&](int u) { return min(lane + u * 32, nvec - 1) * 8; };
    uint8_t* buf = smem_map().work + kTcXOff + warp * (kDepth * kRow) + lane * 16;
    auto request = [&](int rr, int slot) {
        if (rr < rows) {
            const uint8_t* from = reinterpret_cast<const uint8_t*>(op->ptr[0]) + (r0 + rr) * ldx * (kPlanes * 2);
#pragma unroll
            for (int u = 0; u < NPER; ++u)
#pragma unroll
                for (int k = 0; k < kPlanes; ++k) cp_async16(buf + slot * kRow + (u * kPlanes + k) * 512, from + column(u) * (kPlanes * 2) + k * 16, true);
        }
        cp_async_commit();
    };
    int next = warp, slot = 0;
#pragma unroll 1
    for (int d = 0; d < kDepth; ++d, next += kComputeWarps) request(next, d);
#pragma unroll 1
    for (int rr = warp; rr < rows; rr += kComputeWarps, next += kComputeWarps) {
        const long long grp = (r0 + rr) / group;
        Raw8 sc[NPER], sh[NPER];
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            sc[u] = load8_raw(reinterpret_cast<const void*>(op->ptr[4]), grp * op->ld[4] + column(u), op->i[7]);
            sh[u] = load8_raw(reinterpret_cast<const void*>(op->ptr[5]), grp * op->ld[5] + column(u), op->i[8]);
        }
        cp_async_wait<kDepth - 1>();
        const uint8_t* at = buf + slot * kRow;
        auto row = [&](int u, float* f) {
            Vec8<XDT> x;
            x.raw(*reinterpret_cast<const uint4*>(at + u * kPlanes * 512), *reinterpret_cast<const uint4*>(at + u * kPlanes * 512 + (kPlanes - 1) * 512));
            x.get(f);
        };
        float s = 0.f, ss = 0.f;
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            float f[8];
            row(u, f);
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
        const long long out = (r0 + rr) * ldo;
#pragma unroll
        for (int u = 0; u < NPER; ++u) {
            float f[8], g[8], h[8];
            row(u, f);
            unpack8_raw(sc[u], op->i[7], g);
            unpack8_raw(sh[u], op->i[8], h);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = fmaf((f[e] - mean) * rstd, 1.0f + g[e], h[e]);
            if (lane + u * 32 < nvec) put8<ODT>(reinterpret_cast<void*>(op->ptr[1]), out + (lane + u * 32) * 8, f);
        }
        request(next, slot);
        if (++slot == kDepth) slot = 0;
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

// Variant of a norm: x dtype (bits 0-1), fp16 output (bit 2), vectors per lane (bit 3: 8, else 4), gain (bit 4), modulation (bit 5), fewer than
// four rows per scale and shift row (bit 6), rows kept in registers (bit 8)
constexpr int NORM_OWN = 64, NORM_KEEP = 256, NORM_ANY = 128;
__device__ __forceinline__ int norm_variant(const mk_op_desc* op) {
    const int nper = ((op->i[1] >> 3) + 31) / 32;
    const bool w = op->ptr[2] != 0, mod = op->ptr[4] != 0;
    if (op->ptr[3] || (w && mod) || op->i[5] == DT_F32 || nper > (mod ? 4 : 8)) return NORM_ANY;
    return op->i[4] | (op->i[5] == DT_F16 ? 4 : 0) | (nper > 4 ? 8 : 0) | (w ? 16 : 0) | (mod ? 32 : 0) | (mod ? (op->i[6] < 4 ? NORM_OWN : 0) : op->i[3] > (w ? 4 : 1) * kComputeWarps ? NORM_KEEP : 0);
}
template <int V>
__device__ __forceinline__ void op_norm_rows(const mk_op_desc* op, int a0) {
    const int r0 = a0 * op->i[3], rows = min(op->i[3], op->i[0] - r0);
    if constexpr (V == NORM_ANY) norm_two_pass(op, r0, rows);
    else if constexpr ((V & NORM_KEEP) != 0) norm_kept_rows<(V & 8) ? 8 : 4, V & 3, (V & 4) ? DT_F16 : DT_BF16, (V & 16) != 0>(op, r0, rows);
    else if constexpr ((V & NORM_OWN) != 0) norm_own<V & 3, (V & 4) ? DT_F16 : DT_BF16>(op, r0, rows);
    else norm_stream<(V & 8) ? 8 : 4, V & 3, (V & 4) ? DT_F16 : DT_BF16, (V & 16) != 0, (V & 32) != 0>(op, r0, rows);
}

}  // namespace mk
