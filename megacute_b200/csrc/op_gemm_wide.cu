// Translation unit of MK_OP_GEMM with 256 x 256 output tiles on the tcgen05 body (descriptor i 10 = 256 and tensor
// maps attached).  Separate from op_gemm.cu so that each tile shape gets its own register allocation: inlined side
// by side, the wider tile's extra live state spilled registers of the narrow tile's main loop (spills are L2 round
// trips here: batch-64 decode 7 % slower, the MLP block 14 %).
#include "op_gemm_tc_wide.cuh"
#include "ops.cuh"
#include "walk.cuh"

namespace mk {

template <int V>
static __device__ __noinline__ int wide_run(const Params& p, int idx) {
    const SmemMap m = smem_map();
    return run_own_insts(
        p, m.ctrl, idx, [](const mk_op_desc* op) { return is_wide_gemm(op) && wide_variant(op) == V; },
        [&](const mk_op_desc* op, int a0, int a1, int, int seq) -> int {
            op_gemm_tc_wide<V>(p, m.ctrl, m.ring, op, a0, a1, seq);
            return 0;
        },
        [&] { if (threadIdx.x == 0) m.ctrl->wide_uses += 1; });
}

__device__ int mk_run_gemm_wide(const Params& p, int idx) {
    const SmemMap m = smem_map();
    const Meta* mt = &m.ctrl->meta;
    wide_begin_run(m.ctrl);
    for (;;) {
        const int slot = (idx - (int)blockIdx.x) / (int)gridDim.x;
        int last;
        switch (wide_variant(&mt->desc[slot & 1])) {
            case WIDE_PLAIN: last = wide_run<WIDE_PLAIN>(p, idx); break;
            case WIDE_SWIGLU: last = wide_run<WIDE_SWIGLU>(p, idx); break;
            case WIDE_GELU: last = wide_run<WIDE_GELU>(p, idx); break;
            case WIDE_ACT: last = wide_run<WIDE_ACT>(p, idx); break;
            case WIDE_PLAIN + 16: last = wide_run<WIDE_PLAIN + 16>(p, idx); break;
            case WIDE_SWIGLU + 16: last = wide_run<WIDE_SWIGLU + 16>(p, idx); break;
            case WIDE_GELU + 16: last = wide_run<WIDE_GELU + 16>(p, idx); break;
            case WIDE_ACT + 16: last = wide_run<WIDE_ACT + 16>(p, idx); break;
            case WIDE_ANY1: last = wide_run<WIDE_ANY1>(p, idx); break;
            case WIDE_ANY2: last = wide_run<WIDE_ANY2>(p, idx); break;
            case WIDE_GATE1: last = wide_run<WIDE_GATE1>(p, idx); break;
            case WIDE_GATE2: last = wide_run<WIDE_GATE2>(p, idx); break;
            default: last = wide_run<WIDE_ANY0>(p, idx); break;
        }
        if (last < 0) return -1;
        const int next = last + (int)gridDim.x;
        if (!next_is(p, m.ctrl, last, [](const mk_op_desc* op) { return is_wide_gemm(op); })) {
            // (behind the last instruction's barrier: nobody reads the staging rows any more)
            if (threadIdx.x == 0) *(volatile uint32_t*)&m.ctrl->wide_done = m.ctrl->wide_uses;
            return last;
        }
        idx = next;
        stage_following(p, m.ctrl, idx);
    }
}

__device__ void mk_wide_issuer(const Params& p) {
    const SmemMap m = smem_map();
    wide_issuer(p, m.ctrl, m.ring);
}
}  // namespace mk
