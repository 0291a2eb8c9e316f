// Translation unit of MK_OP_GEMM with 256 x 256 output tiles on the tcgen05 body (descriptor i 10 = 256 and tensor
// maps attached).  Separate from op_gemm.cu so that each tile shape gets its own register allocation: inlined side
// by side, the wider tile's extra live state spilled registers of the narrow tile's main loop (spills are L2 round
// trips here: batch-64 decode 7 % slower, the MLP block 14 %).
#include "op_gemm_tc_wide.cuh"
#include "ops.cuh"
#include "walk.cuh"

namespace mk {
__device__ int mk_run_gemm_wide(const Params& p, int idx) {
    const SmemMap m = smem_map();
    wide_begin_run(m.ctrl);
    const int last = run_own_insts(
        p, m.ctrl, idx, [](const mk_op_desc* op) { return is_wide_gemm(op); },
        [&](const mk_op_desc* op, int a0, int a1, int, int seq) -> int {
            op_gemm_tc_wide(p, m.ctrl, m.ring, op, a0, a1, seq);
            return 0;
        },
        [&] { if (threadIdx.x == 0) m.ctrl->wide_uses += 1; });
    // (behind the last instruction's barrier: nobody reads the staging rows any more)
    if (last >= 0 && threadIdx.x == 0) *(volatile uint32_t*)&m.ctrl->wide_done = m.ctrl->wide_uses;
    return last;
}

__device__ void mk_wide_issuer(const Params& p) {
    const SmemMap m = smem_map();
    if ((threadIdx.x & 31) == 0) wide_issuer(p, m.ctrl, m.ring, m.work);
    __syncwarp();
}
}  // namespace mk
