// What the tcgen05 GEMM kernels share: bounded mbarrier waits, bulk copies,
// commits and the parked stores of the epilogue.
#pragma once
#include <cstdint>

#include "kernels.cuh"

namespace ddfmm {

constexpr unsigned long long U_WAIT_NS = 1000000000ull;  // 1 s
constexpr uint32_t U_WAIT_ITERS = 1u << 26;
constexpr int PCH = 32;       // epilogue chunk: complex rows parked per column
constexpr int UPS = PCH + 2;  // parking-area row stride (complex): 16-byte rows, conflict-free 16-byte accesses

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Wait for the phase of parity `parity`; false after limit_ns, 2^26 polls, or
// once *failed is set by another role.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* failed,
                                          unsigned long long limit_ns) {
    const uint32_t addr = smem_u32(bar);
    unsigned long long t0 = 0;
    for (uint32_t it = 0; it < U_WAIT_ITERS; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 255) == 255) {
            if (failed && *failed) return false;
            const unsigned long long t = gtimer();
            if (t0 == 0)
                t0 = t;
            else if (t - t0 > limit_ns)
                return false;
        }
    }
    return false;
}

// mbar_wait by one lane for its warp: polls take shared-memory cycles from the tensor
// core's operand reads.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* failed,
                                          unsigned long long limit_ns) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = !*failed && mbar_wait(bar, parity, failed, limit_ns);
    return __shfl_sync(0xffffffffu, ok, 0);
}

// Whether the phase of this parity has completed; the caller may go on before it looks at
// the answer.
__device__ __forceinline__ uint32_t mbar_peek(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;\n" ::"r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// Epilogue stores of one parked chunk (PCH complex rows from row0 on, 32 columns):
// two columns per instruction, each lane two consecutive rows of one column, as
// one 16-byte store or vector atomic where the output is 16-byte aligned (two
// 8-byte ones otherwise, or one at an odd last row).  Column c of the warp's 32
// writes at Y + (c's yoff) + row.
template <int MODE>
__device__ __forceinline__ void store_one(float2* y, float2 v) {
    if (MODE == GEMM_SET) {
        *y = v;
    } else if (MODE == GEMM_ADD) {
        const float2 o = *y;
        *y = make_float2(o.x + v.x, o.y + v.y);
    } else {
        atomicAdd(y, v);
    }
}
template <int MODE>
__device__ __forceinline__ void store_chunk(const float2* park, float2* Y, long long my_yo, int col_base, int ncol,
                                            int row0, int rows, int lane) {
    const int sub = lane >> 4, r2 = 2 * (lane & 15), i = row0 + r2;
    for (int cc = 0; cc < 32; cc += 2) {
        const int col = cc + sub;
        const long long yb = __shfl_sync(0xffffffffu, my_yo, col);
        if (col_base + cc >= ncol) break;
        if (i >= rows || col_base + col >= ncol) continue;
        const float4 v = *reinterpret_cast<const float4*>(park + col * UPS + r2);
        float2* y = Y + yb + i;
        const bool two = i + 1 < rows;
        if (two && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
            float4* y4 = reinterpret_cast<float4*>(y);
            if (MODE == GEMM_SET) {
                *y4 = v;
            } else if (MODE == GEMM_ADD) {
                const float4 o = *y4;
                *y4 = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
            } else {
                atomicAdd(y4, v);
            }
        } else {
            store_one<MODE>(y, make_float2(v.x, v.y));
            if (two) store_one<MODE>(y + 1, make_float2(v.z, v.w));
        }
    }
}

}  // namespace ddfmm
