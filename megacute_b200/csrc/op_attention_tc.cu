// Translation unit of MK_OP_ATTENTION on tcgen05 (tensor maps attached by the host library), and of the feeder and issuer warps.
#include "op_gemm_tc_wide.cuh"
#include "op_attention_tc.cuh"
#include "ops.cuh"
#include "walk.cuh"

namespace mk {

template <int D>
static __device__ __noinline__ int attention_run(const Params& p, int idx, int slot) {
    const SmemMap m = smem_map();
    at_begin_run(m.ctrl);
    const int last = run_own_insts(
        p, m.ctrl, idx, slot, [](const mk_op_desc* op) { return is_attention_tc(op) && op->i[5] == D; },
        [&](const mk_op_desc* op, int a0, int a1, int a2, int seq) -> int {
            op_attention_tc<D>(p, m.ctrl, op, a0, a1, a2, seq);
            return 0;
        },
        [&] { if (threadIdx.x == 0) m.ctrl->at_turn += 1; });
    // (behind the last instruction's barrier: every product of the run has completed)
    if (D == 128 && last >= 0 && threadIdx.x == 0) mbar_arrive(&m.ctrl->ring_returned);
    return last;
}
__device__ int mk_run_attention(const Params& p, const mk_op_desc* op, int idx, int slot) {
    return op->i[5] == 64 ? attention_run<64>(p, idx, slot) : attention_run<128>(p, idx, slot);
}

__device__ uint32_t mk_feeder(const Params& p) {
    const SmemMap m = smem_map();
    WideFeed wf;
    AtFeed af;
    int run = 0;                                              // what the CTA's previous instruction was: 1 a 256-row tile, head_dim of an attention, 0 neither
    // the whole warp walks the list (and leaves together: the kernel ends with CTA-wide barriers)
    int idx = blockIdx.x;
    for (; idx < p.n_insts; idx += gridDim.x) {
        const Inst in = fetch_inst(p, idx);
        const int opi = in.opi - 1;
        if (opi < 0 || opi >= p.n_ops) break;
        const mk_op_desc* op = p.ops + opi;
        if (is_wide_gemm(op)) {
            if (!wide_feed(p, m.ctrl, m.ring, op, in, run != 1, wf)) break;
            run = 1;
        } else if (is_attention_tc(op)) {
            const int D = op->i[5];
            const bool ok = D == 64 ? at_feed<64>(p, m.ctrl, m.ring, op, in, run != D, af, wf.count) : at_feed<128>(p, m.ctrl, m.ring, op, in, run != D, af, wf.count);
            ++wf.count;
            if (!ok) break;
            run = D;
        } else {
            run = 0;
        }
    }
    if (idx >= p.n_insts) wide_feed_end(m.ctrl, wf);          // (else the CTA is aborting, and so is the issuer)
    return at_feed_left(af);
}

__device__ void mk_feeder_landed(uint32_t left) { at_wait_landed(&smem_map().ctrl->attn, left); }

// The issuer warp runs what the feeder tells it, in order.
__device__ void mk_issuer(const Params& p) {
    const SmemMap m = smem_map();
    Ctrl* c = m.ctrl;
    WideIssue wi;
    AtIssue ai;
    for (uint32_t n = 0;; ++n) {
        if (!issuer_wait(p, c, &c->wide_told[n & 3u], (n >> 2) & 1u, 0, WHERE_DEP, 4)) return;
        const int4 info = c->wide_info[n & 3u];
        if (info.x == 0) return;
        const bool ok = info.x > 0 ? wide_issue(p, c, m.ring, info, wi) : info.y == 64 ? at_issue<64>(p, c, m.ring, info, ai) : at_issue<128>(p, c, m.ring, info, ai);
        if (!ok) return;
    }
}
}  // namespace mk
