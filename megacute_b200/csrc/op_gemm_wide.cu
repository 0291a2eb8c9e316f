// Translation unit of MK_OP_GEMM with output tiles of 256 rows on the tcgen05 body (descriptor i 11 = 256 and tensor
// maps attached).  Separate from op_gemm.cu so that each tile shape gets its own register allocation: inlined side
// by side, the wider tile's extra live state spilled registers of the narrow tile's main loop (spills are L2 round
// trips here: batch-64 decode 7 % slower, the MLP block 14 %).
#include "op_gemm_tc_wide.cuh"
#include "ops.cuh"
#include "walk.cuh"

namespace mk {

template <int V>
static __device__ __noinline__ int wide_run(const Params& p, int idx, int slot) {
    const SmemMap m = smem_map();
    return run_own_insts(
        p, m.ctrl, idx, slot, [](const mk_op_desc* op) { return is_wide_gemm(op) && wide_variant(op) == V; },
        [&](const mk_op_desc* op, int a0, int a1, int, int seq) -> int {
            op_gemm_tc_wide<V>(p, m.ctrl, m.ring, op, a0, a1, seq);
            return 0;
        },
        [&] { if (threadIdx.x == 0) m.ctrl->wide_uses += 1; });
}

// Behind the last instruction of a variant's run: is the CTA's next one of another variant?  (Out of line: so that the registers it needs
// are not saved around the whole run: 88 -> 48 bytes.)
static __device__ __noinline__ bool wide_goes_on(const Params& p, int last, int slot) {
    Ctrl* c = smem_map().ctrl;
    if (next_is(p, c, last, slot, [](const mk_op_desc* op) { return is_wide_gemm(op); })) {
        stage_following(p, c, last + (int)gridDim.x, slot + 1);
        return true;
    }
    // (behind the last instruction's barrier: nobody reads the staging rows any more)
    if (threadIdx.x == 0) {
        __threadfence_block();
        *(volatile uint32_t*)&c->wide_done = c->wide_uses;
    }
    return false;
}

__device__ int mk_run_gemm_wide(const Params& p, int idx, int slot) {
    const SmemMap m = smem_map();
    const Meta* mt = &m.ctrl->meta;
    wide_begin_run(m.ctrl);
    for (;;) {
        int last;
        switch (wide_variant(&mt->desc[slot & 1])) {
#define MK_W(V) case (V): last = wide_run<(V)>(p, idx, slot); break
            MK_W(WIDE_PLAIN); MK_W(WIDE_SWIGLU); MK_W(WIDE_GELU); MK_W(WIDE_ACT);
            MK_W(WIDE_ROPE); MK_W(WIDE_ROPE + 16); MK_W(WIDE_ROPE_T16); MK_W(WIDE_ROPE_T16 + 16);
            MK_W(WIDE_PLAIN + 16); MK_W(WIDE_SWIGLU + 16); MK_W(WIDE_GELU + 16); MK_W(WIDE_ACT + 16);
#define MK_WR(R) MK_W(WIDE_RES + (R)); MK_W(WIDE_RES + ((R) | DT_F32 << 2)); MK_W(WIDE_RES + ((R) | DT_F16 << 2)); \
                 MK_W(WIDE_RES + ((R) | 16)); MK_W(WIDE_RES + ((R) | DT_F32 << 2 | 16)); MK_W(WIDE_RES + ((R) | DT_F16 << 2 | 16))
            MK_WR(DT_BF16); MK_WR(DT_F32); MK_WR(DT_F16);
#undef MK_WR
#undef MK_W
            default: last = wide_run<WIDE_ANY>(p, idx, slot); break;
        }
        if (last < 0) return -1;
        slot += (last - idx) / (int)gridDim.x;                  // (the last instruction's; not Ctrl::run_slot: thread 0 may be in the next run already)
        if (!wide_goes_on(p, last, slot)) return last;
        idx = last + (int)gridDim.x;
        ++slot;
    }
}

}  // namespace mk
