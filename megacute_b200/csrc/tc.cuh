// tcgen05 and tensor-memory helpers shared by the tile GEMMs and the prefill attention.
#pragma once
#include "mk_device.cuh"

namespace mk {

// instruction descriptor, kind::f16: D = f32 (bits 4-5 = 1), A format (bits 7-9) and B format (bits 10-12):
// 0 = fp16, 1 = bf16, both K-major, N = 128 (bits 17-22 = N / 8), M = 128 (bits 24-28 = M / 16).  Both
// operands have one type: bf16, or -- when the activations are runtime-private ones kept in fp16, see
// passes.promote_temps -- fp16, with the packed weight copy converted to fp16 by the host library.
__device__ __forceinline__ uint32_t tc_idesc_n(bool fp16, uint32_t n) {
    const uint32_t fmt = fp16 ? 0u : 1u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ uint32_t tc_idesc(bool fp16) { return tc_idesc_n(fp16, 128); }

// shared-memory matrix descriptor of a K-major tile with the 128-byte swizzle: start address,
// leading byte offset 16 (unused by swizzled K-major layouts), 1024 bytes between 8-row groups,
// descriptor version 1, layout type 2 (128-byte swizzle).  Advancing 16 K-elements inside the
// swizzle atom adds 32 bytes to the start address.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the mbarrier once every tcgen05.mma this thread has issued so far has completed
__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff; selp.u32 %0, 1, 0, q; }" : "=r"(p));
    return p != 0;
}
// 16 consecutive fp32 columns of this thread's lane (warp-wide)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
          "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
}
// 16 columns of this thread's lane, twice
__device__ __forceinline__ void tc_ld16x2(uint32_t ta, uint32_t tb, float* a, float* b) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7]), "=f"(a[8]), "=f"(a[9]),
          "=f"(a[10]), "=f"(a[11]), "=f"(a[12]), "=f"(a[13]), "=f"(a[14]), "=f"(a[15]), "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]),
          "=f"(b[4]), "=f"(b[5]), "=f"(b[6]), "=f"(b[7]), "=f"(b[8]), "=f"(b[9]), "=f"(b[10]), "=f"(b[11]), "=f"(b[12]), "=f"(b[13]),
          "=f"(b[14]), "=f"(b[15])
        : "r"(ta), "r"(tb)
        : "memory");
}
// 32 consecutive fp32 columns of this thread's lane (warp-wide, lanes 32 (warp & 3) .. +31)
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"          // in the same statement: no use of the registers can move above it
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}


__device__ __forceinline__ float4 load4_any(const uint8_t* base, long long elem, int dtype) {
    if (dtype == DT_F32) return __ldcg(reinterpret_cast<const float4*>(base + elem * 4));
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(base + elem * 2));
    if (dtype == DT_F16) {
        const float2 lo = unpack2h(v.x), hi = unpack2h(v.y);
        return make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}
// A thread writes (and, with a residual, reads) whole 32-byte pieces of its own row: whole sectors, as good as 128 bytes of four
// rows at a time, without the detour through shared memory that the operands of the next tile are streaming through (64
// bytes a cycle in, 96 out to the tensor core).  DiT, 32 images: 8.95 -> 8.82 ms together with the prefetch of the residual; what is
// left (4.6 us for 256 x 256 16-bit outputs, 11 with a residual) is the memory system taking the bursts of all SMs at once.
// `whole`: the rows start on 32-byte boundaries; else two 16-byte accesses.
__device__ __forceinline__ void st32B(uint8_t* at, const uint32_t* w, bool whole) {
    if (whole)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                     "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    else {
        reinterpret_cast<uint4*>(at)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(at)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
__device__ __forceinline__ void ld32B(const uint8_t* at, uint32_t* w, bool whole) {
    if (whole)
        asm volatile("ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                     : "l"(at)
                     : "memory");
    else {
        const uint4 a = __ldcg(reinterpret_cast<const uint4*>(at)), b = __ldcg(reinterpret_cast<const uint4*>(at) + 1);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
}
// 16 columns of a row as 16-bit
template <int DT>
__device__ __forceinline__ void put16(uint8_t* at, const float* v, bool whole) {
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = DT == DT_F16 ? pack2h(v[2 * e], v[2 * e + 1]) : pack2(v[2 * e], v[2 * e + 1]);
    st32B(at, w, whole);
}

}  // namespace mk
