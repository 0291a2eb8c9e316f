// Translation unit of the many-sequence form of MK_OP_DECODE_ATTN (compute-warp side; the copies are
// issued by the producer warp, op_gemv_common.cuh).
#define MK_INLINE_WAITS 1
#include "op_decode_bulk.cuh"
#include "ops.cuh"

namespace mk {
// Waits for its own dependencies and publishes its own arrivals.  Returns whether the CTA is aborting.
__device__ bool mk_op_decode_bulk(const Params& p, const mk_op_desc* op, int b, int s, int nwait, int wait_off, int seq,
                                  int narrive, int arrive_off) {
    const SmemMap m = smem_map();
    decode_bulk_body<false>(p, m.ctrl, op, b, 0, s, m.ring, nwait, wait_off, seq);
    return publish(p, m.ctrl, narrive, arrive_off);
}
__device__ bool mk_op_decode_bulk_own(const Params& p, const mk_op_desc* op, int b, int range, int s, int nwait, int wait_off, int seq,
                                      int narrive, int arrive_off) {
    const SmemMap m = smem_map();
    decode_bulk_body<true>(p, m.ctrl, op, b, range, s, m.ring, nwait, wait_off, seq);
    return publish(p, m.ctrl, narrive, arrive_off);
}
}  // namespace mk
