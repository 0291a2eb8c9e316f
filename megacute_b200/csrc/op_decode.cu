// Translation unit of MK_OP_DECODE_ATTN.
#define MK_INLINE_WAITS 1
#include "op_decode.cuh"
#include "ops.cuh"

namespace mk {

template <int D, int GMAX, bool DIRECT>
static __device__ __forceinline__ bool decode_attn(const Params& p, const SmemMap& m, const mk_op_desc* op, int a0, int a1, int a2, int nwait,
                                                   int wait_off, int seq, int narrive, int arrive_off) {
    if (op->i[10] > 1)          // several kv heads per instruction (batched decode)
        return op_decode_attn_heads<D, GMAX, DIRECT>(p, m.ctrl, op, a0, a1, a2, m.work, nwait, wait_off, seq, narrive, arrive_off);
    return op_decode_attn<D, GMAX, DIRECT>(p, m.ctrl, op, a0, a1, a2, m.work, nwait, wait_off, seq, narrive, arrive_off);
}
template <bool DIRECT>
static __device__ __forceinline__ bool decode_attn(const Params& p, const SmemMap& m, const mk_op_desc* op, int a0, int a1, int a2, int nwait,
                                                   int wait_off, int seq, int narrive, int arrive_off) {
    const int G = op->i[1] / op->i[2];
    if (op->i[3] == 64) {
        if (G <= 4) return decode_attn<64, 4, DIRECT>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
        return decode_attn<64, 8, DIRECT>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
    }
    if (G <= 4) return decode_attn<128, 4, DIRECT>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
    return decode_attn<128, 8, DIRECT>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
}

__device__ bool mk_op_decode_attn(const Params& p, const mk_op_desc* op, int a0, int a1, int a2, int nwait, int wait_off,
                                  int seq, int narrive, int arrive_off) {
    const SmemMap m = smem_map();
    if (op->i[11])
        return a1 ? mk_op_decode_bulk_own(p, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off)
                  : mk_op_decode_bulk(p, op, a0, a2, nwait, wait_off, seq, narrive, arrive_off);
    if (op->flags & MK_F_DIRECT_IN) return decode_attn<true>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
    return decode_attn<false>(p, m, op, a0, a1, a2, nwait, wait_off, seq, narrive, arrive_off);
}
}  // namespace mk
