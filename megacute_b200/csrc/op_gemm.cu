// Translation unit of MK_OP_GEMM.
#include "op_gemm.cuh"
#include "op_gemm_tc.cuh"
#include "ops.cuh"
#include "walk.cuh"

namespace mk {
__device__ int mk_run_gemm(const Params& p, int idx, int slot) {
    const SmemMap m = smem_map();
    return run_own_insts(
        p, m.ctrl, idx, slot,
        [](const mk_op_desc* op) { return op->kind == MK_OP_GEMM && op->ptr[11] && !is_wide_gemm(op); },
        // the host library attached tensor maps: tcgen05 body, weights through the producer's ring
        // (the weight tiles have slots and barriers of their own: the ring position is untouched)
        // (tiles of 256 rows have a translation unit of their own, op_gemm_wide.cu: the kernel calls it directly)
        [&](const mk_op_desc* op, int a0, int a1, int a2, int seq) -> int { return op_gemm_tc(p, m.ctrl, m.ring, m.work, op, a0, a1, a2, seq); },
        [&] { tc_next_state(m.ctrl); });
}
// ... and the mma.sync body: a walk of its own, so that its loop over tiles is no part of the other one's registers (frame 204 -> 188 bytes: prompt of
// 333 tokens 1849 -> 1836 us, 64 sequences at context 1024 1528 -> 1526)
__device__ int mk_run_gemm_sync(const Params& p, int idx, int slot) {
    const SmemMap m = smem_map();
    return run_own_insts(
        p, m.ctrl, idx, slot, [](const mk_op_desc* op) { return op->kind == MK_OP_GEMM && !op->ptr[11]; },
        [&](const mk_op_desc* op, int a0, int a1, int a2, int) -> int {
            // (an output tile of 256 rows, i 11, or columns, i 10, is two or four 128 x 128 ones for this body)
            const int mh = op->i[11] == 256 ? 2 : 1, nh = op->i[10] == 256 ? 2 : 1;
            for (int q = 0; q < mh * nh; ++q) {
                const int mt = a0 * mh + q / nh, n = a1 * nh + q % nh;
                if (mt * 128 >= op->i[0]) break;
                // ops with at most 64 activation rows have a single m tile: hold 64 rows and stream deeper
                if (op->i[0] <= 64) {
                    if (op->i[2] % 64 == 0) op_gemm<64, 64, 3>(op, mt, n, a2, m.work);
                    else op_gemm<64, 32, 6>(op, mt, n, a2, m.work);
                } else {
                    op_gemm<128, 32, 4>(op, mt, n, a2, m.work);
                }
            }
            return 0;
        },
        [] {});
}
__device__ void mk_gemm_landed() { wait_x_landed(smem_map().ctrl); }
}  // namespace mk
