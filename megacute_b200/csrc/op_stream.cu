// Translation unit of the ops that stream activations: pointwise tiles and norms of many rows.  Every variant is a function of its
// own around the walk, with the registers it needs: inlined side by side they spill 2 KB per thread.
#include "ops.cuh"
#include "op_stream.cuh"
#include "walk.cuh"

namespace mk {

template <int V>
static __device__ __noinline__ int eltwise_run(const Params& p, int idx, int slot) {
    return run_own_insts(
        p, smem_map().ctrl, idx, slot, [](const mk_op_desc* op) { return op->kind == MK_OP_ELTWISE && ew_variant(op) == V; },
        [](const mk_op_desc* op, int a0, int a1, int, int) -> int {
            op_eltwise<V>(op, a0, a1);
            return 0;
        },
        [] {});
}
template <int V>
static __device__ __noinline__ int norm_run(const Params& p, int idx, int slot) {
    return run_own_insts(
        p, smem_map().ctrl, idx, slot, [](const mk_op_desc* op) { return op->kind == MK_OP_NORM && op->i[3] > 1 && norm_variant(op) == V; },
        [](const mk_op_desc* op, int a0, int, int, int) -> int {
            op_norm_rows<V>(op, a0);
            return 0;
        },
        [] {});
}

__device__ int mk_run_eltwise(const Params& p, const mk_op_desc* op, int idx, int slot) {
    switch (ew_variant(op)) {
#define MK_EW(V) case (V): return eltwise_run<(V)>(p, idx, slot)
        MK_EW(EW_UNARY); MK_EW(EW_BINARY); MK_EW(EW_SWIGLU); MK_EW(EW_MODULATE); MK_EW(EW_GATED);
        MK_EW(EW_UNARY | 16); MK_EW(EW_BINARY | 16); MK_EW(EW_SWIGLU | 16); MK_EW(EW_MODULATE | 16); MK_EW(EW_GATED | 16);
#define MK_ROPE(X, O) MK_EW(EW_ROPE | (X) << 4 | (O) << 6)
        MK_ROPE(DT_BF16, DT_BF16); MK_ROPE(DT_BF16, DT_F16); MK_ROPE(DT_BF16, DT_F32);
        MK_ROPE(DT_F16, DT_BF16); MK_ROPE(DT_F16, DT_F16); MK_ROPE(DT_F16, DT_F32);
        MK_ROPE(DT_F32, DT_BF16); MK_ROPE(DT_F32, DT_F16); MK_ROPE(DT_F32, DT_F32);
#undef MK_ROPE
#undef MK_EW
        default:                                             // (no such variant: the mode or a dtype is not one)
            if (threadIdx.x == 0) report(p, smem_map().ctrl, MK_DEV_BAD_INST, smem_map().ctrl->meta.inst[slot % 3][3].x, 2, op->i[2], idx, 0);
            return -1;
    }
}
__device__ int mk_run_norm(const Params& p, const mk_op_desc* op, int idx, int slot) {
    switch (norm_variant(op)) {
#define MK_N(V) case (V): return norm_run<(V)>(p, idx, slot)
#define MK_NT(V) MK_N((V) | DT_BF16); MK_N((V) | DT_F16); MK_N((V) | DT_F32); MK_N((V) | 4 | DT_BF16); MK_N((V) | 4 | DT_F16); MK_N((V) | 4 | DT_F32)
        MK_NT(0); MK_NT(16); MK_NT(32); MK_NT(32 | NORM_OWN); MK_NT(8); MK_NT(8 | 16);
        MK_NT(NORM_KEEP); MK_NT(NORM_KEEP | 16); MK_NT(NORM_KEEP | 8); MK_NT(NORM_KEEP | 8 | 16);
#undef MK_NT
#undef MK_N
        default: return norm_run<NORM_ANY>(p, idx, slot);
    }
}
}  // namespace mk
