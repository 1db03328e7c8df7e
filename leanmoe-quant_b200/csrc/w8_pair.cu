// W8 rows against the tokens of a prompt (65 and more): the scaled form of the W8 GEMM, on pairs of SMs (tcgen05 cta_group::2).
//
//   y[t, n] = sum_k fp16(scale[n, g(k)] * codes[n, k]) * x[t, k]        (+ resid[t, n], or SwiGLU of two rows)
//
// A cluster of two blocks works on a tile of 256 weight rows (gate/up: 128 gate rows and their 128 up rows) x up to 256 tokens of one
// expert: a block widens 128 of the rows into its own TMEM and fetches half of the tokens, one MMA (M = 256) reads both blocks' halves,
// and each block gets the sums of its own rows.  Persistent, a pair of blocks per pair of SMs; in each block
//   warp 16      TMA: per group of 128 k its 128 code rows (two boxes of 64) and its half of the tokens (two halves of 64 k), swizzled
//   warps 8-15   widen: thread = weight row and half of the group's codes; times the group's scale, rounded to fp16, into TMEM
//   warp 17      of the even block: issues the MMAs (A from TMEM, B from shared memory, D in TMEM over all of k)
//   warps 0-7    collect: the sums out of TMEM, finished, turned over in shared memory for 16-byte stores
// TMEM: D in the first columns (256, or twice the most tokens of a tile if those are fewer than 128; tiles of up to 128 take its halves in
// turn), behind it A of stage s at 64 s: with few tokens a tile there is room for up to six stages.
//
// What bounds it: large tiles the tensor pipe at the clock that the power cap leaves; tiles of 128 tokens and less the widening warps, 900 to 1000
// cycles a group (neither more of them, nor each half of them on groups of its own in turn, nor fewer operations a code changed that).  One block per tile of 256
// rows x 128 tokens (the form before) moved 160 KB through shared memory per 1024 cycles of MMAs (TMA writes, code reads, token reads by the
// MMAs), more than its 128 bytes a clock; a pair moves 96 KB a block, because a block holds half of the tokens only, and widens half as many
// codes per product.  Us of that form / of this one: 50304 x 2048 by 1024 tokens 180 / 144, by 4096 720 / 575 (1.47 PFLOP/s); experts' gate/up at
// 300, 1024 and 4096 tokens 85 / 76, 112 / 89 and 267 / 228, down 50 / 47, 64 / 57 and 152 / 118; 2048 x 2048 by 300 and 1024 tokens 35 / 20 and
// 37 / 25.
//
// Arrivals at the other block's barriers and waits for them are the instructions' default, release and acquire at the scope of a block: they order no
// shared memory between the blocks.  What crosses over is of two other kinds.  TMEM (codes widened, sums taken out) is ordered by tcgen05's fences
// before an arrival and after a wait.  The odd block's tokens are reported to the even block by the TMA itself, which counts their bytes on that block's
// `full`: its widening warps wait for them too, and tell the MMA thread.  Us of gate/up by 300 and 600 tokens and of a prompt of 300 (two layers): the odd
// block's tokens on no barrier of the even block 62.3, 72.3 and 543; on one that the MMA thread waits for besides 64.8, 74.6 and 557, on `a_full` the same; on
// `full` 63.0, 73.1 and 545, and with the addresses of the even block's barriers looked up once, as now, 61.5, 71.4 and 536.  (With
// `.release.cluster` and `.acquire.cluster` on the arrivals instead, every group waited for the memory system: 4096 x 6144 x 2048 168 us, not 94.)
#include "w8_tile.cuh"

#include <algorithm>

namespace lemoq {
namespace {

constexpr int kThreads = 640;                       // five warpgroups: two collect, two widen, the fifth has the TMA warp and the MMA warp
// Registers: 640 threads are launched with 96 each: 61,440, which is 256 x 144 + 256 x 64 + 128 x 64.
constexpr int kRegsCollect = 144, kRegsWiden = 64, kRegsIssue = 64;
constexpr int kTokens = 256;                        // most tokens of a tile
constexpr int kUnit = 32;                           // the MMA's N is a multiple of it
constexpr int kBox = 32;                            // token rows of one TMA box; a last box has 16
constexpr int kStages = 6;                          // at most
constexpr int kCodeBytes = 128 * 128;
constexpr int kRing = 4 * (kCodeBytes + kTokens * 128);  // bytes of all stages
constexpr int kListed = 64;                         // tiles of a pair that are looked up once
constexpr int kTurnWarp = 32 * 64;                  // a collecting warp's 32 tokens x 32 rows (gate/up: 16)
constexpr int kTurn = 8 * kTurnWarp;
constexpr size_t kSmem = kRing + kTurn + 1024;      // + 8 (E + 1) bytes of tile table

__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_slot) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_pair(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}
// D (both blocks) (+)= A (both blocks' TMEM) * B (both blocks' shared memory); one thread of the even block issues; K = 16.
__device__ __forceinline__ void mma_f16_ts_pair(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a),
                 "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u)
                 : "memory");
}
// Arrives on `bar` of both blocks when every MMA this thread has issued so far is complete.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
__device__ __forceinline__ uint32_t at_even_block(uint32_t addr) {
    uint32_t there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(there) : "r"(addr));
    return there;
}
// tma_load_2d into this block's shared memory, completing on a barrier of either block of the pair.
__device__ __forceinline__ void tma_load_2d_at(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar)
                 : "memory");
}
__device__ __forceinline__ void store_at(uint32_t cluster_addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// Of a converged warp, on a barrier of either block.
__device__ __forceinline__ void warp_arrive_at(uint32_t cluster_bar) {
    __syncwarp();
    if (elect_one()) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// 16 lanes x 32 columns: lane l has rows l / 4 (r[4 j], r[4 j + 1]) and 8 + l / 4 (r[4 j + 2], r[4 j + 3]) at columns 8 j + 2 (l mod 4), + 1.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t (&r)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
// Four 8 x 8 matrices of fp16, each turned over: lane l gives the address of row l mod 8 of matrix l / 8.
__device__ __forceinline__ void stmatrix4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Where eight rows of a token lie in the turned tile: eight tokens in a row (what one stmatrix or one quarter of a load touches) are in
// eight different 16-byte banks.
__device__ __forceinline__ uint32_t turned(int token, int piece, bool gate_up) {
    return gate_up ? 32u * token + 16u * (piece ^ ((token >> 2) & 1)) : 64u * token + 16u * (piece ^ ((token >> 1) & 3));
}

// The group scales of one weight row: the thread of the row asks for those of its next tile a tile ahead (a load takes up to three groups
// under load) and takes them one by one off the low end of its registers (up to 16 groups; other rows are read where they are needed).
struct RowScales {
    uint4 ahead[2];
    uint32_t now[8];
    const __half *row, *row_now;
    __device__ __forceinline__ void ask(const W8Shape& p, int e, int wrow) {
        row = p.scale + (static_cast<int64_t>(e) * p.N + min(wrow, p.N - 1)) * (p.K / p.group);
        if (p.scale_vecs > 0) ahead[0] = __ldg(reinterpret_cast<const uint4*>(row));
        if (p.scale_vecs > 1) ahead[1] = __ldg(reinterpret_cast<const uint4*>(row) + 1);
    }
    __device__ __forceinline__ void begin(const W8Shape& p) {
        row_now = row;
#pragma unroll
        for (int v = 0; v < 2; ++v) now[4 * v] = ahead[v].x, now[4 * v + 1] = ahead[v].y, now[4 * v + 2] = ahead[v].z, now[4 * v + 3] = ahead[v].w;
    }
    __device__ __forceinline__ __half next(const W8Shape& p, int g) {
        if (p.scale_vecs == 0) return __ldg(row_now + (p.group == 128 ? g : (g << 7) / p.group));
        const __half h = __ushort_as_half(static_cast<unsigned short>(now[0]));
#pragma unroll
        for (int i = 0; i < 7; ++i) now[i] = __funnelshift_r(now[i], now[i + 1], 16);
        now[7] >>= 16;
        return h;
    }
};

__global__ void __launch_bounds__(kThreads, 1) w8_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                              const __grid_constant__ CUtensorMap map_x16, const W8Shape p) {
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t s_bar[3 * kStages + 5];
    __shared__ int4 s_list[kListed];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ int s_issued;           // stages the block's TMA thread has filled
    __shared__ volatile int s_copies;  // even block: those of the odd block + 1, when that gave up

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage0 = (smem_u32(raw) + 1023u) & ~1023u;
    int* s_first = reinterpret_cast<int*>(raw + (stage0 - smem_u32(raw)) + kRing + kTurn);
    int* s_tok = s_first + p.E + 1;
    const uint32_t bars = smem_u32(s_bar);
    auto full = [&](int s) { return bars + 8u * s; };                    // the stage's copies have landed; even block: both blocks' tokens, odd block: codes only
    auto done = [&](int s) { return bars + 8u * (kStages + s); };        // its MMAs are over: stage and A buffer are free
    auto a_full = [&](int s) { return bars + 8u * (2 * kStages + s); };  // even block: both blocks' codes are widened
    auto d_full = [&](int b) { return bars + 8u * (3 * kStages + b); };
    auto d_free = [&](int b) { return bars + 8u * (3 * kStages + 2 + b); };  // even block: both blocks have taken the sums out
    const uint32_t drained = bars + 8u * (3 * kStages + 4);
    const int rank = blockIdx.x & 1;
    // A stage: the block's codes, then its half of up to `cap` tokens as two halves of 64 k.  As many of them as there are A buffers
    // beside two accumulators of `twice` tokens.
    const int stages = p.stages, twice = min(p.cap, 128);
    const uint32_t half_bytes = 64u * p.cap, stage_bytes = kCodeBytes + 2u * half_bytes, col_a = p.cap > 128 ? 256u : 2u * p.cap;

    if (tid == 0) {
        s_abort = s_copies = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(done(s), 1);
            mbar_init(a_full(s), 16);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(d_full(b), 1);
            mbar_init(d_free(b), 16);
        }
        mbar_init(drained, 1);
        mbar_fence_init();
    }
    if (warp == 17) tmem_alloc_pair(smem_u32(&s_tmem));
    if (tid == 512) {
        tma_prefetch_map(&map_w);
        tma_prefetch_map(&map_x);
        tma_prefetch_map(&map_x16);
    }
    if (p.seg) pdl_wait();  // segments and tokens come from earlier kernels; without segments only the token loads wait
    pdl_trigger();
    const int mt = p.gate_up ? (p.N / 2 + 127) / 128 : (p.N + 255) / 256;
    const int tile0 = blockIdx.x >> 1, stride = gridDim.x >> 1;
    if (warp == 0) {
        fill_tiles(p, p.cap, mt, s_first, s_tok, lane);
        __syncwarp();
        for (int k = lane; k < kListed; k += 32) {
            const Tile t = find_tile(tile0 + k * stride, s_first, s_tok, p.E, p.cap, kUnit);
            s_list[k] = make_int4(t.row0, t.e, t.t0, t.n);
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the barriers of both blocks are there
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int tiles = s_first[p.E], groups = p.K >> 7;
    volatile int* abort = &s_abort;
    const int mine = tile0 < tiles ? (tiles - tile0 + stride - 1) / stride : 0;  // tiles of this pair
    // The rows of this block: two runs of 64 weight rows.  Gate/up: 64 gate rows, then their up rows.
    auto tile = [&](int k) {
        Tile t;
        if (k < kListed) {
            const int4 v = s_list[k];
            t.row0 = v.x, t.e = v.y, t.t0 = v.z, t.n = v.w;
        } else {
            t = find_tile(tile0 + k * stride, s_first, s_tok, p.E, p.cap, kUnit);
        }
        t.row0 = p.gate_up ? t.row0 * 128 + 64 * rank : t.row0 * 256 + 128 * rank;
        t.row1 = p.gate_up ? p.N / 2 + t.row0 : t.row0 + 64;
        return t;
    };

    auto half_of = [&](const Tile& x) { return (x.n + kUnit - 1) / kUnit * (kUnit / 2); };  // tokens of one block

    if (warp >= 16) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == 16) {
        // ---- TMA: one thread ---------------------------------------------------------------------------------------
        if (elect_one()) {
            int s = 0, issued = 0, early = 0;
            uint32_t ph = 1;
            bool ok = true;
            Tile t = tile(0);
            auto stage_at = [&](int k) { return stage0 + static_cast<uint32_t>(k) * stage_bytes; };
            const uint32_t even_full = at_even_block(full(0));  // (full(s) is 8 s behind)
            auto load_codes = [&](const Tile& x, int g, int k) {  // (the odd block's tokens may land before the even block expects them: its arrival is still missing)
                mbar_expect_tx(full(k), kCodeBytes + (rank ? 0u : 4u * half_of(x) * 128u));
                tma_load_2d(stage_at(k), &map_w, g * 128, x.e * p.N + x.row0, full(k));
                tma_load_2d(stage_at(k) + kCodeBytes / 2, &map_w, g * 128, x.e * p.N + x.row1, full(k));
            };
            if (!p.seg) {  // the codes of the first stages do not depend on earlier kernels: on their way while those finish
                if (mine > 0)
                    for (; early < min(stages, groups); ++early) load_codes(t, early, early);
                pdl_wait();
            }
            for (int i = 0; i < mine && ok; ++i) {
                Tile next = t;
                const int half = half_of(t), row = t.t0 + rank * half;
                for (int g = 0; g < groups; ++g) {
                    if (issued >= early) {
                        if (!(ok = thread_wait(done(s), ph, abort))) break;
                        load_codes(t, g, s);
                    }
                    const uint32_t at = stage_at(s) + kCodeBytes, landed = even_full + 8u * s;
                    for (int b = 0; b < half; b += kBox) {
                        const CUtensorMap* map = half - b >= kBox ? &map_x : &map_x16;
                        tma_load_2d_at(at + b * 128, map, g * 128, row + b, landed);
                        tma_load_2d_at(at + half_bytes + b * 128, map, g * 128 + 64, row + b, landed);
                    }
                    ++issued;
                    if (++s == stages) { s = 0; ph ^= 1; }
                    if (g == 0) next = tile(i + 1);
                }
                t = next;
            }
            // the last MMAs' events arrive here before this block may leave
            for (int j = max(0, issued - stages); ok && j < issued; ++j) ok = thread_wait(done(j % stages), (j / stages) & 1, abort);
            if (!ok) {  // gave up: the copies in flight still land in this block's shared memory
                for (int j = max(0, issued - stages); j < issued && mbar_wait(full(j % stages), (j / stages) & 1);) ++j;
            }
            s_issued = issued;
        }
    } else if (warp == 17 && rank == 0) {
        // ---- MMA: one thread of the pair -----------------------------------------------------------------------------
        if (elect_one()) {
            int s = 0, round = 0, before = 0;  // `before`: tokens of the tile before
            uint32_t ph = 0;
            bool ok = true;
            Tile t = tile(0);
            for (int i = 0; i < mine && ok; ++i, ++round) {
                const int n = (t.n + kUnit - 1) / kUnit * kUnit, b = round & 1;
                const uint32_t idesc = idesc_f16(256, n, false), d = tmem + (n <= twice ? static_cast<uint32_t>(twice * b) : 0u);
                // the tile before the last one is out of TMEM, and where one of two neighbours takes both halves so is the last
                if (!(ok = thread_wait(d_free(b), ((round >> 1) & 1) ^ 1, abort))) break;
                if (round > 0 && max(n, before) > twice && !(ok = thread_wait(d_free(b ^ 1), ((round - 1) >> 1) & 1, abort))) break;
                before = n;
                for (int g = 0; g < groups; ++g) {
                    // the widening warps have seen the copies land before they arrive: no wait on full(s) here
                    if (!(ok = thread_wait(a_full(s), ph, abort))) break;
                    tc_fence_after();
                    const uint64_t x0 = smem_desc_sw128(stage0 + static_cast<uint32_t>(s) * stage_bytes + kCodeBytes, 1024);
                    const uint32_t a = tmem + col_a + 64u * s;
#pragma unroll
                    for (int k = 0; k < 8; ++k) mma_f16_ts_pair(d, a + 8u * k, x0 + (k >> 2) * (half_bytes >> 4) + (k & 3) * 2u, idesc, g > 0 || k > 0);
                    tc_commit_pair(done(s));
                    if (g + 1 == groups) tc_commit_pair(d_full(b));
                    if (++s == stages) { s = 0; ph ^= 1; }
                    if (g == 0) t = tile(i + 1);
                }
            }
            if (!ok) {  // gave up: nothing may still write TMEM when it is freed
                tc_commit_pair(drained);
                mbar_wait(drained, 0);
            }
        }
    } else if (warp >= 8 && warp < 16) {
        // ---- widen: thread = weight row, half of the codes of a group ---------------------------------------------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsWiden));
        const int quarter = warp & 3, kh = (warp >> 2) & 1;
        // lane of TMEM -> code row of the stage.  Gate/up: eight gate rows and their eight up rows in every 16 lanes, so that one thread
        // collects both (tmem_ld_16x32).
        const int slot = p.gate_up ? ((lane >> 3) & 1) * 64 + 16 * quarter + 8 * (lane >> 4) + (lane & 7) : 32 * quarter + lane;
        const uint32_t to0 = tmem + (static_cast<uint32_t>(quarter) << 21) + col_a + 32u * kh;
        const uint32_t from0 = stage0 + slot * 128u, swz = slot & 7;
        const uint32_t even_a_full = at_even_block(a_full(0));
        auto weight_row = [&](const Tile& t) { return slot < 64 ? t.row0 + slot : t.row1 + slot - 64; };
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        RowScales sc;
        if (mine > 0) {
            const Tile t = tile(0);
            sc.ask(p, t.e, weight_row(t));
        }
        for (int i = 0; i < mine && ok; ++i) {
            sc.begin(p);
            for (int g = 0; g < groups; ++g) {
                const __half scale = sc.next(p, g);
                // the stage was refilled when its last MMAs were over: its A buffer is free
                if (!(ok = warp_wait(full(s), ph, abort))) break;
                tc_fence_after();
                const uint32_t from = from0 + static_cast<uint32_t>(s) * stage_bytes, to = to0 + 64u * s;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t a[16];
#pragma unroll
                    for (int c = 0; c < 2; ++c) widen16<true>(lds128(from + ((static_cast<uint32_t>(4 * kh + 2 * h + c) ^ swz) << 4)), scale, a + 8 * c);
                    tmem_st16(to + 16u * h, a);
                }
                tmem_wait_st();
                tc_fence_before();
                warp_arrive_at(even_a_full + 8u * s);
                if (++s == stages) { s = 0; ph ^= 1; }
                if (g == 0 && i + 1 < mine) {
                    const Tile t = tile(i + 1);
                    sc.ask(p, t.e, weight_row(t));
                }
            }
        }
    } else if (warp < 8) {
        // ---- collect: warps w and w + 4 take the chunks of 32 tokens of the same 32 lanes in turn ----------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCollect));
        pdl_wait();  // the residual is an earlier kernel's, and y may still be read by one
        const int quarter = warp & 3, odd = warp >> 2;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter) << 21);
        const uint32_t turn = stage0 + kRing + warp * static_cast<uint32_t>(kTurnWarp);
        const bool gu = p.gate_up;
        const int64_t ld = gu ? p.N / 2 : p.N;
        int round = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i, ++round) {
            const Tile t = tile(i);
            const int n = (t.n + kUnit - 1) / kUnit * kUnit, b = round & 1;
            const uint32_t d = lanes + (n <= twice ? static_cast<uint32_t>(twice * b) : 0u);
            if (!(ok = warp_wait(d_full(b), (round >> 1) & 1, abort))) break;
            tc_fence_after();
            uint32_t out[4][4][4];  // [chunk][eight tokens][rows 0-7, 8-15, 16-23, 24-31; gate/up: rows 0-7, 8-15]
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (32 * (2 * c + odd) < n) {
                    uint32_t lo[16], hi[16];
                    tmem_ld_16x32(lo, d + 32u * (2 * c + odd));
                    tmem_ld_16x32(hi, d + 32u * (2 * c + odd) + (16u << 16));
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float f[8];
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            f[v] = __uint_as_float(lo[4 * j + v]);
                            f[4 + v] = __uint_as_float(hi[4 * j + v]);
                        }
                        if (gu) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                float y0, y1;
                                swiglu2(f[4 * h], f[4 * h + 2], f[4 * h + 1], f[4 * h + 3], y0, y1);
                                out[c][j][h] = pack_half2(y0, y1);
                            }
                        } else {
#pragma unroll
                            for (int h = 0; h < 4; ++h) out[c][j][h] = pack_half2(f[2 * h], f[2 * h + 1]);
                        }
                    }
                }
            }
            tc_fence_before();
            warp_arrive_at(at_even_block(d_free(b)));  // everything has left TMEM: a later tile may begin
            // turned over in shared memory, a lane stores eight rows of a token
            const int row = t.row0 + (gu ? 16 : 32) * quarter, lim = gu ? p.N / 2 : p.N;
            __half* y = p.y + static_cast<int64_t>(t.t0) * ld;
            const __half* res = p.resid ? p.resid + static_cast<int64_t>(t.t0) * ld : nullptr;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int tok0 = 32 * (2 * c + odd);
                if (tok0 < t.n) {
                    __syncwarp();
                    if (gu) {
#pragma unroll
                        for (int j = 0; j < 4; j += 2)
                            stmatrix4_t(turn + turned(8 * (j + (lane >> 4)) + (lane & 7), (lane >> 3) & 1, true), out[c][j][0], out[c][j][1], out[c][j + 1][0],
                                        out[c][j + 1][1]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            stmatrix4_t(turn + turned(8 * j + (lane & 7), lane >> 3, false), out[c][j][0], out[c][j][1], out[c][j][2], out[c][j][3]);
                    }
                    __syncwarp();
                    if (p.wide) {
                        const int pieces = gu ? 2 : 4, shift = gu ? 1 : 2, piece = lane & (pieces - 1), at = row + 8 * piece;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int j = k * (32 >> shift) + (lane >> shift);
                            if (j < 32 && tok0 + j < t.n && at < lim) {
                                uint4 v = lds128(turn + turned(j, piece, gu));
                                if (res) {
                                    const uint4 r4 = __ldcg(reinterpret_cast<const uint4*>(res + (tok0 + j) * ld + at));
                                    __half2* vh = reinterpret_cast<__half2*>(&v);
                                    const __half2* rh = reinterpret_cast<const __half2*>(&r4);
#pragma unroll
                                    for (int e = 0; e < 4; ++e) vh[e] = __hadd2(vh[e], rh[e]);
                                }
                                *reinterpret_cast<uint4*>(y + (tok0 + j) * ld + at) = v;
                            }
                        }
                    } else {
                        const int at = row + lane;
                        if (lane < (gu ? 16 : 32) && at < lim) {
                            for (int j = 0; j < 32 && tok0 + j < t.n; ++j) {
                                unsigned short u;
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(turn + turned(j, lane >> 3, gu) + 2u * (lane & 7)));
                                __half v = __ushort_as_half(u);
                                if (res) v = __hadd(v, res[(tok0 + j) * ld + at]);
                                y[(tok0 + j) * ld + at] = v;
                            }
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0 && s_abort) {
        if (p.err_flag) atomicOr(p.err_flag, LEMOQ_FLAG_WAIT_TIMEOUT);
        if (rank) store_at(at_even_block(smem_u32(const_cast<int*>(&s_copies))), s_issued + 1);
    }
    cluster_sync();  // the other block's arrivals and MMAs are over
    if (rank ? s_abort : s_copies) {  // the odd block gave up: it stays until the even block has seen its last tokens land
        if (rank == 0 && tid == 0) {
            const int there = s_copies - 1;
            for (int j = max(0, there - stages); j < there; ++j) {
                if (j >= s_issued) mbar_expect_tx(full(j % stages), 2u * half_of(tile(j / groups)) * 128u);  // (this block gave up earlier)
                if (!mbar_wait(full(j % stages), (j / stages) & 1)) break;
            }
        }
        cluster_sync();
    }
    if (warp == 17) {
        tc_fence_after();
        tmem_free_pair(tmem);
    }
}

}  // namespace

int launch_w8_pair(W8Shape p, const __half* x, const int8_t* codes, const LaunchCfg& lc) {
    CUtensorMap map_w, map_x, map_x16;
    if (int rc = encode_rows_map(&map_w, codes, 1, static_cast<int64_t>(p.E) * p.N, p.K, 64)) return rc;
    if (int rc = encode_rows_map(&map_x, x, 2, p.T, p.K, kBox)) return rc;
    if (int rc = encode_rows_map(&map_x16, x, 2, p.T, p.K, 16)) return rc;
    const int gk = p.K / p.group, pairs = std::max(1, sm_count() / 2);
    p.wide = (p.gate_up ? p.N / 2 : p.N) % 8 == 0 && aligned16(p.y) && aligned16(p.resid);
    p.scale_vecs = aligned16(p.scale) && p.group == 128 && (gk == 8 || gk == 16) ? gk / 8 : 0;
    const int64_t mt = p.gate_up ? (p.N / 2 + 127) / 128 : (p.N + 255) / 256;
    // Tokens of a tile.  One segment: cut so that the rounds of the pairs cost least; by the cycles that were measured a group costs
    // 700 + 1.6 n and a tile 1000 + 8 n beside (2048 rows x 512 tokens: 25 us with tiles of 256 tokens on 16 pairs, 20.5 with 64 on 64; 50304 x 512:
    // 102 with 128 in 11 rounds, 85 with 256 in 6).  Experts: nearly all of them in one tile (a second one widens the codes again).
    p.cap = kTokens;
    int64_t most = 0;  // tiles, at most
    if (p.seg) {
        const int64_t mean = (p.T + p.E - 1) / p.E;
        while (p.cap > 2 * kUnit && 4 * (p.cap - kUnit) >= 5 * mean) p.cap -= kUnit;
        most = mt * (p.T / p.cap + std::min<int64_t>(p.E, p.T));
    } else {
        int64_t least = INT64_MAX;
        for (int cap = kTokens; cap >= 2 * kUnit; cap -= kUnit) {
            const int64_t tiles = mt * ((p.T + cap - 1) / cap), cost = (tiles + pairs - 1) / pairs * ((700 + 8 * cap / 5) * (p.K >> 7) + 1000 + 8 * cap);
            if (cost < least) {
                least = cost;
                p.cap = cap;
                most = tiles;
            }
        }
    }
    p.stages = p.cap > 128 ? 4 : std::min(kStages, (512 - 2 * p.cap) / 64);
    const size_t smem = kSmem + 8 * (static_cast<size_t>(p.E) + 1);
    if (int rc = allow_smem(w8_pair_kernel, smem)) return rc;
    LaunchCfg pair = lc;
    pair.cluster = 2;
    const int grid = 2 * static_cast<int>(std::min<int64_t>(pairs, std::max<int64_t>(most, 1)));
    return launch_kernel(w8_pair_kernel, dim3(grid), dim3(kThreads), smem, pair, map_w, map_x, map_x16, p);
}

}  // namespace lemoq
