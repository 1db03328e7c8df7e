// Attention of a prompt over the fp16 cache: row t sees slots [0, pos[t]] (head_dim 128), tcgen05 for both products.
//
// One block = one head x 256 query rows (few blocks: 128), as two tiles of 128 that take turns: while the warpgroup of one tile is in its softmax,
// the tensor pipe works for the other.  Per 128 cache slots and tile:
//   S = Q K^T   A, B from shared memory, 128 x 128 fp32 in TMEM
//   softmax     one thread per row, in base 2: its row in registers, maximum, exp2, fp16, back into TMEM over S
//   PV          A = the fp16 weights from TMEM, B = V (d is the contiguous side: MN-major), 128 x 128 fp32 in TMEM
//   O           accumulates in TMEM.  The maximum a row's weights are taken against follows the true one only when that has grown by more
//               than 2^8 (the weights stay below 256, the sum of them in fp32): then, which is rare after the first steps, O is rescaled.
// Blocks are handed out longest first.  No S x S matrix exists anywhere.  (Two query tiles taking turns, sums in TMEM and rescaling only
// beyond a slack are the published method of FlashAttention-4.)
//
// Bounded by exp2 (16 per SM and clock: 2048 cycles for the two tiles of a step) and the MMAs (2048 cycles as well), which the two tiles
// overlap.  (With O in registers, 128 of them beside a row of S, the kernel spilled: 412 us at 4096 rows and 16 heads
// instead of 111.)
#include "prompt.h"
#include "tc.cuh"

namespace lemoq {
namespace {

constexpr int kThreads = 320;     // two softmax warpgroups, the TMA warp, the MMA warp
constexpr float kSlack = 8.f;     // log2 of how far the true maximum may run ahead of the one in use
constexpr int kRows = 128;        // query rows of a tile
constexpr int kSlots = 128;       // cache slots of a step
constexpr int kHalf = 128 * 128;  // bytes of 128 rows x 64 values
constexpr int kTile = 2 * kHalf;
constexpr int kKvStages = 2;
constexpr size_t kSmem = static_cast<size_t>(2 * kTile + 2 * kKvStages * kTile) + 1024;

struct AttnShape {
    const int64_t* pos;
    __half* out;
    int T, heads, S, tiles;  // tiles: of a block, 1 or 2
    float scale_log2;
    int* err_flag;
};

// 2^x, 0 below 2^-126 (exp2f would keep those, for three more instructions an element)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__global__ void __launch_bounds__(kThreads, 1) prompt_attn_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                  const __grid_constant__ CUtensorMap map_v, const AttnShape p) {
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t s_bar[16];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ int s_most[2];  // last slot any row of the tile sees

    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t q_smem = (smem_u32(raw) + 1023u) & ~1023u, k_smem = q_smem + 2 * kTile, v_smem = k_smem + kKvStages * kTile;
    const uint32_t bars = smem_u32(s_bar);
    const uint32_t q_full = bars;
    auto k_full = [&](int s) { return bars + 8u * (1 + s); };
    auto k_free = [&](int s) { return bars + 8u * (3 + s); };
    auto v_full = [&](int s) { return bars + 8u * (5 + s); };
    auto v_free = [&](int s) { return bars + 8u * (7 + s); };
    auto s_full = [&](int i) { return bars + 8u * (9 + i); };
    auto p_full = [&](int i) { return bars + 8u * (11 + i); };
    auto o_full = [&](int i) { return bars + 8u * (13 + i); };
    const uint32_t drained = bars + 8u * 15;
    const int head = blockIdx.y, t0 = (gridDim.x - 1 - blockIdx.x) * p.tiles * kRows;  // the last rows see most: they start first
    volatile int* abort = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        s_most[0] = s_most[1] = 0;
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full(i), 1);
            mbar_init(k_free(i), 1);
            mbar_init(v_full(i), 1);
            mbar_init(v_free(i), 1);
            mbar_init(s_full(i), 1);
            mbar_init(p_full(i), 4);
            mbar_init(o_full(i), 1);
        }
        mbar_init(drained, 1);
        mbar_fence_init();
    }
    if (warp == 9) tmem_alloc(smem_u32(&s_tmem), 512);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    int my_pos = -1;  // rows behind the end see nothing
    if (warp < 4 * p.tiles && t0 + tid < p.T) {
        const int64_t q = p.pos[t0 + tid];
        my_pos = static_cast<int>(q < 0 ? 0 : (q >= p.S ? p.S - 1 : q));
        atomicMax(&s_most[warp >> 2], my_pos);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int live = p.tiles == 2 && t0 + kRows < p.T ? 2 : 1;
    const int steps = max(s_most[0], s_most[1]) / kSlots + 1;  // both tiles run over the same slots

    if (warp == 8) {
        if (elect_one()) {
            mbar_expect_tx(q_full, live * kTile);
            for (int i = 0; i < live; ++i)
                for (int c = 0; c < 2; ++c) tma_load_2d(q_smem + i * kTile + c * kHalf, &map_q, head * 128 + 64 * c, t0 + i * kRows, q_full);
            bool ok = true;
            int j = 0;
            for (; j < steps; ++j) {
                const int s = j % kKvStages;
                const uint32_t ph = ((j / kKvStages) & 1) ^ 1;
                const int row = head * p.S + j * kSlots;
                if (!(ok = thread_wait(k_free(s), ph, abort))) break;
                mbar_expect_tx(k_full(s), kTile);
                for (int c = 0; c < 2; ++c) tma_load_2d(k_smem + s * kTile + c * kHalf, &map_k, 64 * c, row, k_full(s));
                if (!(ok = thread_wait(v_free(s), ph, abort))) {
                    mbar_wait(k_full(s), (j / kKvStages) & 1);
                    break;
                }
                mbar_expect_tx(v_full(s), kTile);
                for (int c = 0; c < 2; ++c) tma_load_2d(v_smem + s * kTile + c * kHalf, &map_v, 64 * c, row, v_full(s));
            }
            if (!ok) {  // gave up: the copies in flight still land in this block's shared memory
                mbar_wait(q_full, 0);
                for (int i = max(0, j - kKvStages); i < j; ++i) {
                    mbar_wait(k_full(i % kKvStages), (i / kKvStages) & 1);
                    mbar_wait(v_full(i % kKvStages), (i / kKvStages) & 1);
                }
            }
        }
    } else if (warp == 9) {
        if (elect_one()) {
            const uint32_t id_s = idesc_f16(128, 128, false), id_o = idesc_f16(128, 128, true);
            bool ok = thread_wait(q_full, 0, abort);
            // S of tile i, step j; P of the same tile overwrites it, and MMAs of one thread run in order
            auto scores = [&](int i, int s) {
                const uint64_t a = smem_desc_sw128(q_smem + i * kTile, 1024), b = smem_desc_sw128(k_smem + s * kTile, 1024);
#pragma unroll
                for (int k = 0; k < 8; ++k) mma_f16_ss(tmem + 128u * i, a + (k >> 2) * (kHalf >> 4) + (k & 3) * 2u, b + (k >> 2) * (kHalf >> 4) + (k & 3) * 2u, id_s, k != 0);
                tc_commit(s_full(i));
            };
            if (ok && (ok = thread_wait(k_full(0), 0, abort))) {
                tc_fence_after();
                for (int i = 0; i < live; ++i) scores(i, 0);
                tc_commit(k_free(0));
            }
            for (int j = 0; j < steps && ok; ++j) {
                const int s = j % kKvStages, sn = (j + 1) % kKvStages;
                if (!(ok = thread_wait(v_full(s), (j / kKvStages) & 1, abort))) break;
                if (j + 1 < steps && !(ok = thread_wait(k_full(sn), ((j + 1) / kKvStages) & 1, abort))) break;
                for (int i = 0; i < live && ok; ++i) {
                    if (!(ok = thread_wait(p_full(i), j & 1, abort))) break;
                    tc_fence_after();
                    const uint64_t v = smem_desc_sw128(v_smem + s * kTile, 1024, kHalf);
#pragma unroll
                    for (int k = 0; k < 8; ++k) mma_f16_ts(tmem + 256u + 128u * i, tmem + 128u * i + 8u * k, v + k * (16u * 128u >> 4), id_o, j > 0 || k > 0);
                    tc_commit(o_full(i));
                    if (j + 1 < steps) scores(i, sn);
                }
                if (!ok) break;
                tc_commit(v_free(s));
                if (j + 1 < steps) tc_commit(k_free(sn));
            }
            if (!ok) {  // gave up: nothing may still write TMEM when it is freed
                tc_commit(drained);
                mbar_wait(drained, 0);
            }
        }
    } else if (warp >> 2 < live) {
        const int i = warp >> 2;
        const uint32_t lanes = static_cast<uint32_t>(warp & 3) << 21;
        const uint32_t s_at = tmem + lanes + 128u * i, o_at = tmem + lanes + 256u + 128u * i;
        float m = -INFINITY, l = 0.f;  // the maximum in use (times the scale, in base 2)
        bool ok = true;
        for (int j = 0; j < steps; ++j) {
            if (!(ok = warp_wait(s_full(i), j & 1, abort))) break;
            tc_fence_after();
            const int seen = my_pos - j * kSlots;  // slots [0, seen] of this step are visible
            const bool all = __all_sync(0xffffffffu, seen >= kSlots - 1);
            uint32_t r[4][32];  // the row stays in registers for both passes
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(r[c], s_at + 32 * c);
            tmem_wait_ld();
            if (!all) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int d = 0; d < 32; ++d)
                        if (32 * c + d > seen) r[c][d] = 0xff800000u;  // -inf: weight 0
            }
            float tops[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tops[c] = __uint_as_float(r[c][0]);
#pragma unroll
                for (int d = 1; d < 31; d += 2) tops[c] = fmaxf(fmaxf(tops[c], __uint_as_float(r[c][d])), __uint_as_float(r[c][d + 1]));
                tops[c] = fmaxf(tops[c], __uint_as_float(r[c][31]));
            }
            const float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
            const float m_new = fmaxf(m, top * p.scale_log2);
            const bool grown = m_new > m + kSlack;  // the first visible slot of a row always is
            if (__any_sync(0xffffffffu, grown)) {
                const float alpha = grown ? exp2f(m - m_new) : 1.f;
                if (grown) m = m_new;
                l *= alpha;
                if (j > 0) {
                    if (!(ok = warp_wait(o_full(i), (j - 1) & 1, abort))) break;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 128; c += 16) {
                        uint32_t v[16];
                        tmem_ld16(v, o_at + c);
                        tmem_wait_ld();
#pragma unroll
                        for (int d = 0; d < 16; ++d) v[d] = __float_as_uint(__uint_as_float(v[d]) * alpha);
                        tmem_st16(o_at + c, v);
                    }
                }
            }
            const float shift = m > -INFINITY ? m : 0.f;
            float sums[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t w[16];
#pragma unroll
                for (int d = 0; d < 32; d += 2) {
                    const float e0 = ex2(fmaf(__uint_as_float(r[c][d]), p.scale_log2, -shift)), e1 = ex2(fmaf(__uint_as_float(r[c][d + 1]), p.scale_log2, -shift));
                    sums[d & 2] += e0;
                    sums[(d & 2) + 1] += e1;
                    const __half2 h = __floats2half2_rn(e0, e1);
                    w[d / 2] = *reinterpret_cast<const uint32_t*>(&h);
                }
                tmem_st16(s_at + 16 * c, w);  // over columns this thread has read
            }
            l += (sums[0] + sums[1]) + (sums[2] + sums[3]);
            tmem_wait_st();
            tc_fence_before();
            warp_arrive(p_full(i));
        }
        if (ok && (ok = warp_wait(o_full(i), (steps - 1) & 1, abort))) {
            tc_fence_after();
            const float inv = 1.f / l;
            __half* dst = p.out + (static_cast<int64_t>(t0 + tid) * p.heads + head) * 128;
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
                uint32_t r[32];
                tmem_ld32(r, o_at + c);
                tmem_wait_ld();
                if (t0 + tid < p.T) {
#pragma unroll
                    for (int e = 0; e < 32; e += 8) {
                        __align__(16) __half h[8];
#pragma unroll
                        for (int d = 0; d < 8; ++d) h[d] = __float2half_rn(__uint_as_float(r[e + d]) * inv);
                        *reinterpret_cast<uint4*>(dst + c + e) = *reinterpret_cast<const uint4*>(h);
                    }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (tid == 0 && s_abort && p.err_flag) atomicOr(p.err_flag, LEMOQ_FLAG_WAIT_TIMEOUT);
    if (warp == 9) {
        tc_fence_after();
        tmem_free(tmem, 512);
    }
}

}  // namespace

int launch_prompt_attn(const PromptAttn& a, const LaunchCfg& lc) {
    CUtensorMap map_q, map_k, map_v;
    const int64_t width = static_cast<int64_t>(a.heads) * 128;
    if (int rc = encode_rows_map(&map_q, a.q, 2, a.T, width, kRows)) return rc;
    if (int rc = encode_rows_map(&map_k, a.keys, 2, static_cast<int64_t>(a.heads) * a.S, 128, kSlots)) return rc;
    if (int rc = encode_rows_map(&map_v, a.values, 2, static_cast<int64_t>(a.heads) * a.S, 128, kSlots)) return rc;
    const cudaError_t err = cudaFuncSetAttribute(prompt_attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
    if (err != cudaSuccess) return set_error(LEMOQ_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(err));
    AttnShape p;
    p.pos = a.pos; p.out = a.out; p.T = a.T; p.heads = a.heads; p.S = a.S;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.err_flag = a.err_flag;
    // One tile a block while every such block has an SM of its own: the pair shares the SM's exp2 unit, which is idle elsewhere (us of four layers of
    // a prompt with two tiles a block / one: 512 tokens 965 / 945, 1024 1251 / 1237; 1500 tokens, 192 tiles, 1510 / 1530, 4096 3820 / 4100).
    p.tiles = static_cast<int64_t>((a.T + kRows - 1) / kRows) * a.heads <= sm_count() ? 1 : 2;
    return launch_kernel(prompt_attn_kernel, dim3((a.T + p.tiles * kRows - 1) / (p.tiles * kRows), a.heads), dim3(kThreads), kSmem, lc, map_q, map_k, map_v, p);
}

}  // namespace lemoq
