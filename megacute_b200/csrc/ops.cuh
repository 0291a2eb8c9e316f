// Entry points of the op bodies.  Every op body lives in its own translation unit and the library
// is built as relocatable device code: measured on sm_100a, when the bodies share one translation
// unit with the kernel, ptxas' whole-program register allocation spills the inner loop of the
// streaming linear to local memory (with 227 KB of the SM given to shared memory almost no L1 is
// left, so each spill is an L2 round trip: 6x slower), however the calls are arranged.  Compiled
// separately, each body gets its own allocation under a cap of 168 registers (12 warps of
// 168 fill the SM's register file).
//
// All take the op descriptor and the instruction's arguments by value and find the CTA's shared
// memory through the kernel's dynamic shared-memory window.
#pragma once
#include "mk_device.cuh"

namespace mk {

// ring position in / out is packed as stage | phase << 8
// (this op waits for its own dependencies and publishes its own arrivals; returns -1 when aborting)
__device__ int mk_op_gemv_units(const Params& p, const mk_op_desc* op, int o0, int o1, int seq, int packed_pos, int nwait,
                                int wait_off, int narrive, int arrive_off);
// (the same when x is a direct operand)
__device__ int mk_op_gemv_direct(const Params& p, const mk_op_desc* op, int o0, int o1, int seq, int packed_pos, int nwait,
                                 int wait_off, int narrive, int arrive_off);
// body of the finisher warp (op_gemv_mma.cuh): runs until the CTA's instruction list ends
__device__ void mk_gemv_finisher(const Params& p);
__device__ int mk_op_gemv_general(const Params& p, const mk_op_desc* op, int o0, int o1, int seq, int packed_pos);
// Tile GEMM.  The kernel's loop has fetched instruction `idx`, the CTA's `slot`-th, and chosen this body; the body runs it and every
// following instruction of the CTA that is its own (walk.cuh), waiting for the dependencies and publishing the
// arrivals of each itself (begin_op says why).  Returns the index of the last instruction executed, -1 when the CTA is
// aborting.  (The ring position is untouched: the weight tiles have slots of their own.)
__device__ int mk_run_gemm(const Params& p, int idx, int slot);
// (the same for ops without tensor maps: mma.sync body)
__device__ int mk_run_gemm_sync(const Params& p, int idx, int slot);
// (abort path: its activation tiles still in flight have landed)
__device__ void mk_gemm_landed();
// (the same with output tiles of 256 rows; only for ops the host library bound to the tcgen05 body)
__device__ int mk_run_gemm_wide(const Params& p, int idx, int slot);
// body of the issuer warp: the MMAs of every tile GEMM with 256-row tiles and of every tcgen05 attention, until the feeder warp says that the list has ended
__device__ void mk_issuer(const Params& p);
__device__ void mk_op_attention(const mk_op_desc* op, int a0, int a1, int a2);
// (the tcgen05 body, for ops the host library attached tensor maps to: like mk_run_gemm, for runs of one head_dim)
__device__ int mk_run_attention(const Params& p, const mk_op_desc* op, int idx, int slot);
// body of the feeder warp: walks the CTA's instruction list and requests the tiles of every prefill attention bound to the
// tcgen05 body and the activation tiles of every tile GEMM with 256-row tiles; runs until the list ends or the CTA aborts.
// Returns what mk_feeder_landed, on the abort path, waits for: the attention's tiles still in flight.  (Half a stage of a 256-row tile,
// requested without the weights' half, cannot be waited for: the pause behind it covers that.)
__device__ uint32_t mk_feeder(const Params& p);
__device__ void mk_feeder_landed(uint32_t left);
// (waits for its own dependencies and publishes its own arrivals; returns whether the CTA is aborting)
__device__ bool mk_op_decode_attn(const Params& p, const mk_op_desc* op, int a0, int a1, int a2, int nwait, int wait_off,
                                  int seq, int narrive, int arrive_off);
// (many-sequence form: all kv heads of a sequence per instruction, whole cache rows through bulk copies)
__device__ bool mk_op_decode_bulk(const Params& p, const mk_op_desc* op, int b, int s, int nwait, int wait_off, int seq,
                                  int narrive, int arrive_off);
__device__ bool mk_op_decode_bulk_own(const Params& p, const mk_op_desc* op, int b, int range, int s, int nwait, int wait_off, int seq,
                                      int narrive, int arrive_off);
// pointwise tiles and norms with several rows per instruction (op_stream.cuh): like mk_run_gemm, for runs of their own kind
__device__ int mk_run_eltwise(const Params& p, const mk_op_desc* op, int idx, int slot);
__device__ int mk_run_norm(const Params& p, const mk_op_desc* op, int idx, int slot);
// finalize / norm of one row / rope_append / increment / gather / argmax; returns false for an unknown kind
__device__ bool mk_op_pointwise(const mk_op_desc* op, int a0, int a1, long long direct_off);

struct SmemMap {
    uint8_t* ring;
    uint8_t* work;
    Ctrl* ctrl;
};
__device__ __forceinline__ SmemMap smem_map() {
    extern __shared__ __align__(1024) uint8_t mk_smem[];
    SmemMap m;
    m.ring = mk_smem;
    m.work = mk_smem + kRingBytes;
    m.ctrl = reinterpret_cast<Ctrl*>(mk_smem + kRingBytes + kWorkBytes);
    return m;
}

}  // namespace mk
