// Decode attention over the int8 mirror on the tensor cores (head_dim 128): one query row per head, any number of heads
// (batch x heads act as heads), split-KV.
//
// The codes go from memory to the tensor core without passing a register: TMA lands tiles of 128 positions, tcgen05.mma
// kind::i8 reads them where they are.  Both products are integer and exact; what is not int8 travels as three 7-bit digits:
//   S[pos]  = K (128 pos x 128 d, A, K-major) x the digits of q (B, 3 of 16 columns)        thread = position
//   O[d]    = V^T (128 d x 128 pos, A, MN-major) x the digits of p * v_scale (B)            thread = head dimension
// A softmax warp owns 32 positions, which is one k-step of the second product: its digits have columns 3w .. 3w + 2 to
// themselves and are zero for the other warps' positions.  So every warp keeps a running maximum of its own, and no barrier
// joins the four inside the loop; they are merged when the block is done.
//
//   warp 4  TMA       warp 5  MMA       warps 0-3  scores, exp2, digits; collect the weighted values
//
// Bounded by HBM with many heads (two blocks per SM, three tiles of 32 KB each in flight); by the chain TMA - S - softmax - O
// (about 1 us a tile) with few.  The kernel this replaces for int8 spent 7 instructions on every code: 169 us for 64 x 16 heads x
// 2049 positions (3.2 TB/s).
#include "tc.cuh"

#include <algorithm>

namespace lemoq {
namespace {

constexpr int kThreads = 192;
constexpr int kStages = 3;
constexpr int kPos = 128;                  // positions of a tile
constexpr int kTileBytes = kPos * 128;
constexpr int kDigits = 16 * 128;          // a B operand: 16 rows of 128 bytes, swizzled
constexpr size_t kSmem = static_cast<size_t>(kStages) * 2 * kTileBytes + 4 * kDigits + 1024;
constexpr int kMerge = 20;                 // splits of a head that are merged from registers (at most 32)
constexpr int kAhead = 4;                  // tiles a position's scales are loaded ahead
constexpr uint32_t kTmemCols = 64;         // S at 0 and 16, O at 32 and 48

struct Shape {
    const __half* q;
    const __half *ks, *vs;
    const int32_t* filled;
    __half* out;
    float* part;
    unsigned int* counters;
    int* err_flag;
    int heads, S, splits;
    float scale_log2;
};

// address of byte k of row r of a B operand
__device__ __forceinline__ uint32_t digit_at(uint32_t base, int r, int k) { return base + r * 128 + ((((k >> 4) ^ (r & 7)) << 4) | (k & 15)); }
__device__ __forceinline__ void sts_u8(uint32_t addr, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_digits(uint32_t base, int row, int k, int x) {
    sts_u8(digit_at(base, row, k), x & 0x7f);
    sts_u8(digit_at(base, row + 1, k), (x >> 7) & 0x7f);
    sts_u8(digit_at(base, row + 2, k), (x >> 14) & 0xff);
}
__device__ __forceinline__ float digits_f32(uint32_t d0, uint32_t d1, uint32_t d2) {
    return fmaf(16384.f, static_cast<float>(static_cast<int>(d2)), fmaf(128.f, static_cast<float>(static_cast<int>(d1)), static_cast<float>(static_cast<int>(d0))));
}

// Work item i: (head, split).  Every head has the same filled length, so a split has the same tiles in every head; at most the
// splits asked for are used, none of them empty (but for an empty cache).
struct Items {
    int splits, all_tiles, per, count;
    __device__ __forceinline__ int first(int i) const { return (i % splits) * per; }
    __device__ __forceinline__ int tiles(int i) const { return min(per, all_tiles - first(i)); }
};
// A place in the block's sequence of tiles.
struct Cursor {
    int i, t, j;  // item, tile of the item, tiles so far
    __device__ __forceinline__ void next(const Items& w) {
        ++j;
        if (++t == w.tiles(i)) {
            t = 0;
            i += gridDim.x;
        }
    }
};

// Dimension tid of a head from its splits (maximum, sum, values), in split order.  Everything of the first kMerge comes in one trip to L2, a
// maximum and a sum in a lane each.  Us a call without / with it, mean of 20 calls in a graph on the same cache (on caches from memory): 16 heads x 1025
// positions 7.7 / 6.9 (8.4 / 7.5), 2049 8.4 / 7.4 (9.9 / 8.9), 4097 in 19 splits 9.5 / 8.5 (11.2 / 10.2); 8 heads x 4097 in 37 splits, seventeen of
// them one after the other, 10.1 / 9.4 (11.6 / 10.8); 256 to 1024 heads, which have no splits, the same.  (A function of its own: inlined, its
// registers made the tiles' loop slower, 1.5 us a layer of a lockstep step of five sequences.)
__device__ __noinline__ float merged(const float* parts, int splits, int tid) {
    const int lane = tid & 31;
    const bool mine = lane < min(splits, kMerge);
    const float pm = mine ? __ldcg(parts + lane * 130) : -INFINITY, pl = mine ? __ldcg(parts + lane * 130 + 1) : 0.f;
    float pv[kMerge], num = 0.f, den = 0.f;
#pragma unroll
    for (int x = 0; x < kMerge; ++x)
        if (x < splits) pv[x] = __ldcg(parts + x * 130 + 2 + tid);
    float top = warp_max(pm);
    for (int x = kMerge; x < splits; ++x) top = fmaxf(top, __ldcg(parts + x * 130));
    const float pf = exp2f(pm - top);
#pragma unroll
    for (int x = 0; x < kMerge; ++x) {
        if (x < splits) {
            num = fmaf(pv[x], __shfl_sync(0xffffffffu, pf, x), num);
            den = fmaf(__shfl_sync(0xffffffffu, pl, x), __shfl_sync(0xffffffffu, pf, x), den);
        }
    }
    for (int x = kMerge; x < splits; ++x) {
        const float f = exp2f(__ldcg(parts + x * 130) - top);
        num = fmaf(__ldcg(parts + x * 130 + 2 + tid), f, num);
        den = fmaf(__ldcg(parts + x * 130 + 1), f, den);
    }
    return num / den;
}

__global__ void __launch_bounds__(kThreads, 2) attn_i8_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const Shape p) {
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t s_bar[2 * kStages + 10];
    __shared__ float2 s_step[4][4];       // [step & 3][warp]: rescale of the warp's running sums, scale of its digits; a warp can be two steps ahead
    __shared__ float s_m[2][4], s_l[2][4];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ int s_last;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t tiles_at = (smem_u32(raw) + 1023u) & ~1023u, digits_at = tiles_at + kStages * 2 * kTileBytes;
    auto q_at = [&](int b) { return digits_at + kDigits * b; };
    auto p_at = [&](int b) { return digits_at + kDigits * (2 + b); };
    const uint32_t bars = smem_u32(s_bar);
    auto full = [&](int s) { return bars + 8u * s; };
    auto freed = [&](int s) { return bars + 8u * (kStages + s); };
    auto s_full = [&](int b) { return bars + 8u * (2 * kStages + b); };
    auto o_full = [&](int b) { return bars + 8u * (2 * kStages + 2 + b); };
    auto p_full = [&](int b) { return bars + 8u * (2 * kStages + 4 + b); };
    auto q_full = [&](int b) { return bars + 8u * (2 * kStages + 6 + b); };
    const uint32_t drained = bars + 8u * (2 * kStages + 8), joined = drained + 8u;
    volatile int* abort = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(freed(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(s_full(b), 1);
            mbar_init(o_full(b), 1);
            mbar_init(p_full(b), 4);
            mbar_init(q_full(b), 1);
        }
        mbar_init(drained, 1);
        mbar_init(joined, 4);
        mbar_fence_init();
    }
    if (warp == 5) tmem_alloc(smem_u32(&s_tmem), kTmemCols);
    for (uint32_t i = tid * 16; i < 4 * kDigits; i += kThreads * 16) asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(digits_at + i), "r"(0) : "memory");
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_wait();
    pdl_trigger();

    int n = *p.filled;
    if (n < 0 || n > p.S) {
        if (p.err_flag && tid == 0) atomicOr(p.err_flag, LEMOQ_FLAG_BAD_LENGTH);
        n = n < 0 ? 0 : p.S;
    }
    Items w;
    w.all_tiles = (n + kPos - 1) / kPos;
    w.per = max(1, (w.all_tiles + p.splits - 1) / p.splits);
    w.splits = max(1, (w.all_tiles + w.per - 1) / w.per);
    w.count = n > 0 ? p.heads * w.splits : 0;
    if (n == 0)
        for (int i = blockIdx.x; i < p.heads; i += gridDim.x)
            if (tid < 128) p.out[static_cast<int64_t>(i) * 128 + tid] = __float2half_rn(0.f);

    if (warp == 4) {
        if (elect_one()) {
            bool ok = true;
            Cursor c{static_cast<int>(blockIdx.x), 0, 0};
            for (; c.i < w.count; c.next(w)) {
                const int s = c.j % kStages, row = (c.i / w.splits) * p.S + (w.first(c.i) + c.t) * kPos;
                if (!(ok = thread_wait(freed(s), ((c.j / kStages) & 1) ^ 1, abort))) break;
                mbar_expect_tx(full(s), 2 * kTileBytes);
                tma_load_2d(tiles_at + s * 2 * kTileBytes, &map_k, 0, row, full(s));
                tma_load_2d(tiles_at + s * 2 * kTileBytes + kTileBytes, &map_v, 0, row, full(s));
            }
            if (!ok) {  // gave up: the copies in flight still land in this block's shared memory
                for (int j = max(0, c.j - kStages); j < c.j; ++j) mbar_wait(full(j % kStages), (j / kStages) & 1);
            }
        }
    } else if (warp == 5) {
        if (elect_one()) {
            const uint32_t id_s = idesc_i8(128, 16, false), id_o = idesc_i8(128, 16, true);
            Cursor ahead{static_cast<int>(blockIdx.x), 0, 0}, c = ahead;
            // scores of the next tile; its buffer was read before the weights of the tile before the last were handed over
            auto scores = [&]() {
                const int round = (ahead.i - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x), j = ahead.j, s = j % kStages;
                if (ahead.t == 0 && !thread_wait(q_full(round & 1), (round >> 1) & 1, abort)) return false;
                if (!thread_wait(full(s), (j / kStages) & 1, abort)) return false;
                tc_fence_after();
                const uint64_t k_desc = smem_desc_sw128(tiles_at + s * 2 * kTileBytes, 1024), q_desc = smem_desc_sw128(q_at(round & 1), 1024);
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_i8_ss(tmem + 16u * (j & 1), k_desc + 2 * k, q_desc + 2 * k, id_s, k != 0);
                tc_commit(s_full(j & 1));
                ahead.next(w);
                return true;
            };
            bool ok = ahead.i >= w.count || scores();
            for (; ok && c.i < w.count; c.next(w)) {
                if (ahead.i < w.count && !(ok = scores())) break;
                const int j = c.j, s = j % kStages;
                if (!(ok = thread_wait(p_full(j & 1), (j >> 1) & 1, abort))) break;
                tc_fence_after();
                const uint64_t v_desc = smem_desc_sw128(tiles_at + s * 2 * kTileBytes + kTileBytes, 1024), p_desc = smem_desc_sw128(p_at(j & 1), 1024);
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_i8_ss(tmem + 32u + 16u * (j & 1), v_desc + k * (32u * 128u >> 4), p_desc + 2 * k, id_o, k != 0);
                tc_commit(o_full(j & 1));
                tc_commit(freed(s));
            }
            if (!ok) {  // gave up: nothing may still write TMEM when it is freed
                tc_commit(drained);
                mbar_wait(drained, 0);
            }
        }
    } else {
        const uint32_t lanes = static_cast<uint32_t>(warp) << 21;
        float o[4] = {0.f, 0.f, 0.f, 0.f};  // o[x]: dimension tid over the positions of warp x
        bool ok = true;
        auto take = [&](int j) {
            if (!warp_wait(o_full(j & 1), (j >> 1) & 1, abort)) return false;
            tc_fence_after();
            uint32_t r[16];
            tmem_ld16(r, tmem + lanes + 32u + 16u * (j & 1));
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float2 c = s_step[j & 3][x];
                o[x] = fmaf(o[x], c.x, digits_f32(r[3 * x], r[3 * x + 1], r[3 * x + 2]) * c.y);
            }
            tc_fence_before();
            return true;
        };
        // Loads are asked for long before they are used (under load one takes as long as three tiles): the query of an item two
        // items ahead, the scales of a position kAhead tiles ahead, across items.
        auto query_row = [&](int i) {
            return i < w.count ? __ldcg(reinterpret_cast<const uint2*>(p.q + static_cast<int64_t>(i / w.splits) * 128 + 4 * lane)) : make_uint2(0, 0);
        };
        auto query_digits = [&](const uint2& v, int round) {  // every warp finds the scale, warp 0 writes the digits
            const __half* h = reinterpret_cast<const __half*>(&v);
            float f[4], sx, inv;
            uint32_t top = 0;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                f[x] = __half2float(h[x]);
                top = max(top, __float_as_uint(fabsf(f[x])));
            }
            digit_scale(__reduce_max_sync(0xffffffffu, top), sx, inv);
            if (warp == 0) {
#pragma unroll
                for (int x = 0; x < 4; ++x) sts_digits(q_at(round & 1), 0, 4 * lane + x, digit_round(f[x], inv));
                fence_async_smem();
                warp_arrive(q_full(round & 1));
            }
            return sx * p.scale_log2;
        };
        __half k_ring[kAhead], v_ring[kAhead];
        Cursor c{static_cast<int>(blockIdx.x), 0, 0}, far = c;
        auto scales = [&](__half& k, __half& v) {
            if (far.i >= w.count) return;
            const int pos = (w.first(far.i) + far.t) * kPos + tid;
            if (pos < n) {
                const int64_t at = static_cast<int64_t>(far.i / w.splits) * p.S + pos;
                k = __ldcg(p.ks + at);
                v = __ldcg(p.vs + at);
            }
            far.next(w);
        };
        uint32_t joins = 0;
        auto join = [&]() {  // the four softmax warps (an mbarrier: a named barrier has no limit)
            warp_arrive(joined);
            return warp_wait(joined, joins++ & 1, abort);
        };
        int round = 0;
        uint2 q_next = query_row(c.i);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            k_ring[u] = v_ring[u] = __half();
            scales(k_ring[u], v_ring[u]);
        }
        float sx_q = 0.f, sx_next = c.i < w.count ? query_digits(q_next, 0) : 0.f, m = -INFINITY, l = 0.f;
        q_next = query_row(c.i + gridDim.x);
        while (ok && c.i < w.count) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (!ok || c.i >= w.count) break;
                const int i = c.i, t = c.t, j = c.j, tiles = w.tiles(i);
                if (t == 0) {
                    sx_q = sx_next;
                    if (i + static_cast<int>(gridDim.x) < w.count) sx_next = query_digits(q_next, round + 1);
                    q_next = query_row(i + 2 * gridDim.x);
                    m = -INFINITY;
                    l = 0.f;
#pragma unroll
                    for (int x = 0; x < 4; ++x) o[x] = 0.f;
                }
                if (!(ok = warp_wait(s_full(j & 1), (j >> 1) & 1, abort))) break;
                tc_fence_after();
                uint32_t r[4];
                tmem_ld4(r, tmem + lanes + 16u * (j & 1));
                tmem_wait_ld();
                const bool in = (w.first(i) + t) * kPos + tid < n;
                const float s = in ? digits_f32(r[0], r[1], r[2]) * sx_q * __half2float(k_ring[u]) : -INFINITY;
                const float m_new = fmaxf(m, warp_max(s)), base = m_new > -INFINITY ? m_new : 0.f;
                const float alpha = exp2f(m - base), e = exp2f(s - base), ev = in ? e * __half2float(v_ring[u]) : 0.f;
                scales(k_ring[u], v_ring[u]);
                l = fmaf(l, alpha, e);
                m = m_new;
                float sx, inv;
                digit_scale(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(ev))), sx, inv);
                // the sums of the tile before the last leave TMEM; its digits' buffer is free then
                if (t > 1 && !(ok = take(j - 2))) break;
                if (lane == 0) s_step[j & 3][warp] = make_float2(alpha, sx);
                sts_digits(p_at(j & 1), 3 * warp, tid, digit_round(ev, inv));
                fence_async_smem();
                tc_fence_before();
                warp_arrive(p_full(j & 1));
                c.next(w);
                if (t + 1 < tiles) continue;

                // the item is done: the last two tiles' sums, then the four warps side by side
                if ((t > 0 && !(ok = take(j - 1))) || !(ok = take(j))) break;
                ++round;
                l = warp_sum(l);
                if (lane == 0) {
                    s_m[round & 1][warp] = m;
                    s_l[round & 1][warp] = l;
                }
                if (!(ok = join())) break;
                const float* sm = s_m[round & 1];
                const float big = fmaxf(fmaxf(sm[0], sm[1]), fmaxf(sm[2], sm[3]));
                float acc = 0.f, sum = 0.f;
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float f = exp2f(sm[x] - big);
                    acc = fmaf(o[x], f, acc);
                    sum = fmaf(s_l[round & 1][x], f, sum);
                }
                const int head = i / w.splits;
                __half* out = p.out + static_cast<int64_t>(head) * 128 + tid;
                if (w.splits == 1) {
                    *out = __float2half_rn(acc / sum);
                    continue;
                }
                float* parts = p.part + static_cast<int64_t>(head) * p.splits * 130;
                float* part = parts + (i % w.splits) * 130;
                part[2 + tid] = acc;
                if (tid == 0) {
                    part[0] = big;
                    part[1] = sum;
                }
                // the last split of the head merges them in split order
                __threadfence();
                if (!(ok = join())) break;
                if (tid == 0) s_last = atomicAdd(p.counters + head, 1u) == static_cast<unsigned int>(w.splits) - 1u;
                if (!(ok = join())) break;
                if (!s_last) continue;
                __threadfence();
                *out = __float2half_rn(merged(parts, w.splits, tid));
                if (tid == 0) p.counters[head] = 0u;
            }
        }
        if (!ok) {  // gave up: the counters are left as a finished launch leaves them
            for (int i = c.i; i < w.count; i += gridDim.x)
                if (tid == 0) p.counters[i / w.splits] = 0u;
        }
    }
    __syncthreads();
    if (tid == 0 && s_abort && p.err_flag) atomicOr(p.err_flag, LEMOQ_FLAG_WAIT_TIMEOUT);
    if (warp == 5) {
        tc_fence_after();
        tmem_free(tmem, kTmemCols);
    }
}

}  // namespace

// (The query is read eight bytes at a time; one that starts elsewhere takes the split kernel, which reads it by element.)
bool attn_i8_eligible(const AttnParams& p) {
    return p.D == 128 && p.kv_head_stride == static_cast<int64_t>(p.S) * 128 && static_cast<int64_t>(p.heads) * p.S <= 0x7fffffff && p.heads <= 65535 &&
           (reinterpret_cast<uintptr_t>(p.q) & 7u) == 0;
}

int launch_attn_i8(const AttnParams& a, const LaunchCfg& lc) {
    CUtensorMap map_k, map_v;
    const int64_t rows = static_cast<int64_t>(a.heads) * a.S;
    if (int rc = encode_rows_map(&map_k, a.k, 1, rows, 128, kPos)) return rc;
    if (int rc = encode_rows_map(&map_v, a.v, 1, rows, 128, kPos)) return rc;
    const cudaError_t err = cudaFuncSetAttribute(attn_i8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem));
    if (err != cudaSuccess) return set_error(LEMOQ_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(err));
    Shape p;
    p.q = a.q; p.ks = a.ks; p.vs = a.vs; p.filled = a.filled; p.out = a.out; p.part = a.part; p.counters = a.counters; p.err_flag = a.err_flag;
    // num_splits is the most a caller wants.  With a head for every SM a split is not worth its partial sums, also where half of the two
    // places an SM has stay empty (us with 1 / 2 / 3 / 4 splits, cold caches):
    //   160 heads    700 positions 16 / 25 / 23 / 23    2048: 29 / 37 / 33 / 37    4096: 47 / 59 / 49 / 55
    //   240 heads    700 positions 20 / 25 / 29 / 29    2048: 35 / 41 / 45 / 45    4096: 59 / 64 / 68 / 70
    //   512 heads    700 positions 31 / 41 / 47 / 49    2048: 62 / 72 / 76 / 76    4096: 102 / 115 / 119 / 117
    // The exceptions are small: 148 heads x 4096 45 / 43 / 47 / 47, 320 (a third round of items) x 4096 92 / 88 / 86 / 84.
    p.heads = a.heads; p.S = a.S; p.splits = a.heads >= sm_count() ? 1 : a.num_splits; p.scale_log2 = a.qk_scale_log2;
    const int64_t items = static_cast<int64_t>(a.heads) * p.splits;
    return launch_kernel(attn_i8_kernel, dim3(static_cast<unsigned>(std::min<int64_t>(items, 2 * sm_count()))), dim3(kThreads), kSmem, lc, map_k, map_v, p);
}

}  // namespace lemoq
