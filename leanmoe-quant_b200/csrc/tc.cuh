// tcgen05 / TMEM / TMA primitives of the tensor-core kernels (sm_100a).  The mbarrier primitives are in stream.cuh.
#pragma once

#include <cuda.h>  // CUtensorMap (types only: the encoder is looked up at run time)

#include "kernels.h"
#include "stream.cuh"

namespace lemoq {

// ---- TMA ---------------------------------------------------------------------------------------------------------
// 2-D tiled load into shared memory, completing on an mbarrier.  c0 (the inner coordinate) times the element size must
// be a multiple of 16 bytes; rows outside the tensor are filled with zeros.  Local memory only, no multicast.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(c0), "r"(c1), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Power-of-two scale of a group of fp32 values and its inverse: |x| / scale < 2^20, so x is three 7-bit digits
// d2 * 2^14 + d1 * 2^7 + d0 (fp16 values within 2^9 of the maximum are exact, the rest good to 2^-20 of it).  `top`: the largest of the
// absolute values' bit patterns, in whose order NaN and infinity come last; digits cannot express those, so the scale is NaN then.
__device__ __forceinline__ void digit_scale(uint32_t top, float& sx, float& inv) {
    const int e = static_cast<int>(top >> 23);  // biased exponent
    const int k = e > 20 ? e - 19 : 2;  // zero or denormal range: a fixed tiny scale keeps the arithmetic exact
    sx = e == 255 ? __uint_as_float(0x7fffffffu) : __uint_as_float(static_cast<uint32_t>(k) << 23);
    inv = __uint_as_float(static_cast<uint32_t>(254 - k) << 23);
}
__device__ __forceinline__ int digit_round(float x, float inv) {  // round to nearest even, |x| * inv < 2^20
    return static_cast<int>(__float_as_uint(fmaf(x, inv, 12582912.0f)) - 0x4B400000u);
}

// One arrival for the warp.
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if (elect_one()) mbar_arrive(bar);
}

// Row-major (rows, cols) matrix of 1- or 2-byte elements as a tensor map with 128-byte swizzle; the box is box_rows rows of
// 128 bytes.  `base` 16-byte aligned, cols * element size a multiple of 16.
int encode_rows_map(CUtensorMap* map, const void* base, int elem_bytes, int64_t rows, int64_t cols, int box_rows);

// ---- tcgen05 -----------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Arrives on `bar` when every tcgen05.mma this thread has issued so far is complete.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Instruction descriptor of kind::f16 with fp16 operands and fp32 accumulators: M x N, A K-major, B K- or MN-major.
__device__ __forceinline__ constexpr uint32_t idesc_f16(int m, int n, bool b_mn_major) {
    return (1u << 4) | (b_mn_major ? 1u << 16 : 0u) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
// Shared-memory descriptor of a tile in the 128-byte swizzled layout TMA writes (rows of 128 bytes, atoms of 8 rows).
// K-major: sbo = bytes between groups of 8 rows.  MN-major: sbo = bytes between groups of 8 k, lbo = between 64-element blocks.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr, uint32_t sbo, uint32_t lbo = 16) {
    return static_cast<uint64_t>((addr & 0x3ffffu) >> 4) | (static_cast<uint64_t>(lbo >> 4) << 16) | (static_cast<uint64_t>(sbo >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// D[tmem] (+)= A[tmem] * B[smem], one thread issues; K = 16.
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a),
                 "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
                 : "memory");
}
// D[tmem] (+)= A[smem] * B[smem].
__device__ __forceinline__ void mma_f16_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a),
                 "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
                 : "memory");
}

// Instruction descriptor of kind::i8 with signed operands and int32 accumulators: M x N, B K-major, A K- or MN-major.  K = 32.
__device__ __forceinline__ constexpr uint32_t idesc_i8(int m, int n, bool a_mn_major) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (a_mn_major ? 1u << 15 : 0u) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
__device__ __forceinline__ void mma_i8_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a),
                 "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
                 : "memory");
}
// Shared-memory stores of this thread become visible to the tensor core (async proxy) once it has also arrived somewhere.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Warp w of a warpgroup reads / writes lanes [32 w, 32 w + 32) of TMEM, one lane per thread, n consecutive 32-bit columns.
__device__ __forceinline__ void tmem_ld4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_ld32(uint32_t (&r)[32], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
        "%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
        "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of one thread; `abort` as below.
__device__ __forceinline__ bool thread_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
    if (mbar_test(bar, parity)) return true;
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && *abort) return false;
    }
    *abort = 1;
    return false;
}
// Bounded wait of a whole warp: the same outcome in every lane.  `abort` is a flag in shared memory: a warp that gave up
// sets it, and every later wait in the block ends at once.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
    bool ok = mbar_try_wait(bar, parity);
    if (__all_sync(0xffffffffu, ok)) return true;
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        if ((i & 1023u) == 1023u && __any_sync(0xffffffffu, *abort)) break;
        ok = ok || mbar_try_wait(bar, parity);
        if (__all_sync(0xffffffffu, ok)) return true;
    }
    *abort = 1;
    return false;
}

}  // namespace lemoq
