// Device helpers of the tensor-core kernels: mbarriers with bounded waits, shared-memory matrix descriptors, commits,
// bulk copies, and the tensor-map encoder looked up through the runtime.
#pragma once

#include <cuda.h>

#include "swlm_internal.h"

namespace swlm {

constexpr int kTcSpinLimit = 1 << 22;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// Bounded wait on phase parity; returns false when the limit was reached. The loop is two instructions per
// attempt (try_wait suspends the warp for a while by itself): waiting warps share their scheduler with warps
// that still dequantise.
#define SWLM_MBAR_WAIT(SEM)                                                            \
    asm volatile(                                                                      \
        "{\n\t"                                                                        \
        ".reg .pred p, q;\n\t"                                                         \
        ".reg .u32 n;\n\t"                                                             \
        "mov.u32 n, 0;\n\t"                                                            \
        "mbarrier.test_wait.parity" SEM ".shared::cta.b64 p, [%1], %2;\n\t"            \
        "@p bra SWLM_DONE;\n\t"                                                        \
        "SWLM_TRY:\n\t"                                                                \
        "mbarrier.try_wait.parity" SEM ".shared::cta.b64 p, [%1], %2;\n\t"             \
        "@p bra SWLM_DONE;\n\t"                                                        \
        "add.u32 n, n, 1;\n\t"                                                         \
        "setp.lt.u32 q, n, %3;\n\t"                                                    \
        "@q bra SWLM_TRY;\n\t"                                                         \
        "SWLM_DONE:\n\t"                                                               \
        "selp.u32 %0, 1, 0, p;\n\t"                                                    \
        "}"                                                                            \
        : "=r"(done) : "r"(addr), "r"(parity), "r"((unsigned)kTcSpinLimit) : "memory")
__device__ __forceinline__ bool mbar_wait_addr(unsigned addr, unsigned parity) {
    unsigned done;
    SWLM_MBAR_WAIT("");
    return done != 0;
}
// The same where threads of another CTA of the cluster arrive.
__device__ __forceinline__ bool mbar_wait_cluster_addr(unsigned addr, unsigned parity) {
    unsigned done;
    SWLM_MBAR_WAIT(".acquire.cluster");
    return done != 0;
}
#undef SWLM_MBAR_WAIT
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) { return mbar_wait_addr(smem_u32(bar), parity); }

// The same for a converged warp: all its lanes get the same answer, also when some of them saw the limit.
__device__ __forceinline__ bool mbar_wait_warp(unsigned addr, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait_addr(addr, parity)); }
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long* bar, unsigned parity) { return mbar_wait_warp(smem_u32(bar), parity); }
__device__ __forceinline__ bool mbar_wait_cluster_warp(unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait_cluster_addr(smem_u32(bar), parity)); }

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024
// bytes apart (stride byte offset); leading byte offset unused for this layout; descriptor version 1.
// Its low word holds the address, the high one is constant: places 32 bytes apart along K differ by 2, a tile `bytes` further on by
// bytes / 16. Put together where it is used, so that a loop over the MMAs of a step adds 32-bit numbers only.
__device__ __forceinline__ unsigned umma_desc_lo(unsigned smem_addr) { return (smem_addr & 0x3FFFFu) >> 4; }
constexpr unsigned kUmmaDescHi = (1024u >> 4) | 1u << 14 | 2u << 29;

// One lane of a converged warp, the same one every time: the MMAs of a warp that runs its loop as a whole are issued by it. (A loop
// inside `if (lane == 0)` spends 60 to 100 clocks per MMA on moving operands to uniform registers.)
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One tile of a 2-D tensor map (x = innermost coordinate), completion counted on an mbarrier of this CTA.
__device__ __forceinline__ void tma_load_2d(unsigned smem_dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_dst), "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
// The same where the mbarrier (a cluster address) may lie in the other CTA of a pair.
__device__ __forceinline__ void tma_load_2d_pair(unsigned smem_dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_dst), "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
// `bytes` contiguous bytes (16-byte aligned, a multiple of 16) into shared memory.
__device__ __forceinline__ void bulk_load(unsigned smem_dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// cuTensorMapEncodeTiled, looked up through the runtime so that the library does not link against the driver
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encode_fn() {
    static TensorMapEncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(f);
    }();
    return fn;
}

// 4 / x of x >= 1, infinity included: the unit's reciprocal (one unit in the last place) and one step of Newton's iteration, without a
// branch (a division's slow path is one, behind which a lane's independent values would be worked out one after the other: 6 % of a
// prompt). Times four, because the reciprocal of a large x is subnormal, which the unit takes for zero.
__device__ __forceinline__ float four_over(float x) {
    const float q = 0.25f * x;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
    const float refined = fmaf(r, fmaf(-q, r, 1.0f), r);
    return q < INFINITY ? refined : 0.0f;
}

}  // namespace swlm
