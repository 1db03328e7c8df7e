// W8 rows against many tokens on the tensor cores: prompts (thousands of tokens), batches of tens, and the routed experts
// of both (tokens sorted by expert, a segment per expert).
//
//   y[t, n] = sum_g scale[n, g] * ( sum_{k in group g} codes[n, k] * x[t, k] )        (+ resid[t, n], or SwiGLU of two rows)
//
// The weight rows are the M side of tcgen05.mma (128 rows a tile, lane = row), the tokens the N side: an expert with nine
// tokens costs an N of 16 and not a tile of 128.  Two forms:
//   exact   here, up to 64 tokens a tile.  int8 codes are exact in fp16, so the products are those of the integer kernels: the codes
//           are widened, not scaled.  The fp32 sum of one group of 128 codes leaves TMEM, is scaled in fp32 and added to
//           the row's accumulators in registers.
//   scaled  more tokens, for prompts: w8_pair.cu.
//
// One persistent block per SM, a tile = two M tiles (256 weight rows; for gate/up 128 gate rows and their 128 up rows)
// x up to NT tokens of one expert:
//   warp 16      TMA: per group of 128 k the codes (2 x 128 rows x 128 bytes) and the tokens (two halves of 64 k), swizzled
//   warps 8-15   a warpgroup per M tile, thread = weight row: widen the codes of a group into TMEM (two buffers)
//   warps 17, 18 issue the MMAs, one warp per M tile: A = widened codes from TMEM, B = tokens from shared memory, D in TMEM
//   warps 0-7    a warpgroup per M tile, thread = weight row: collect the sums (per group / at the end), finish the rows
// TMEM: D of tile w, buffer b at column 128 w + 64 b, A of tile w, buffer b at 256 + 128 w + 64 b.
//
// What bounds it: with few tokens per expert the bytes of the codes (HBM).  A in TMEM instead of shared memory, because widened
// codes in shared memory would add a write and a read of twice the codes' size.  Widening and collecting are different warps
// because either is a chain of waits, and the TMA and MMA loops are one thread each because a vote after every wait cost
// that warp 160 cycles (NT = 16: 3200 cycles per group with both by the same warps and `lane == 0` issue, 1700 with
// separate warps and elect.sync).  One MMA thread for both tiles left the tensor pipe idle for a quarter of the time (a wait
// that is over costs it 200 cycles): with two, one waits while the other's MMAs run.
#include "w8_tile.cuh"

#include <algorithm>
#include <mutex>

namespace lemoq {

int encode_rows_map(CUtensorMap* map, const void* base, int elem_bytes, int64_t rows, int64_t cols, int box_rows) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) == cudaSuccess &&
            found == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<Encode>(fn);
    });
    if (!encode) return set_error(LEMOQ_ERR_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * elem_bytes};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem_bytes), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    // 256-byte promotion: a box is 128 bytes of each row, and the next one along the rows comes soon.  With 128 the experts of 64 tokens took 73.8 and
    // 43.0 us (gate/up, down), with 256 69.7 and 39.9.
    const CUresult rc = encode(map, elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims,
                               strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return set_error(LEMOQ_ERR_CUDA, "cuTensorMapEncodeTiled: error %d", static_cast<int>(rc));
    return LEMOQ_OK;
}

namespace {

constexpr int kThreads = 640;       // five warpgroups: two collect, two widen, the fifth has the TMA warp and the MMA warp
// Registers: 640 threads are launched with 96 each (61,440); 256 x 144 + 256 x 56 + 128 x 72 = 60,416 afterwards.
constexpr int kExactTokens = 64;    // most tokens of a tile
constexpr int kRegsCollect = 144, kRegsWiden = 56, kRegsIssue = 72;
constexpr int kTileRows = 256;      // weight rows of a tile (two M tiles of 128)
constexpr int kCodeBytes = 2 * 128 * 128;
constexpr int kScaleStride = 36;    // bytes of a row's group scales in shared memory: 16 of them and a pad against bank conflicts
constexpr uint32_t kColA = 256;     // first TMEM column of the widened codes

template <int NT>
struct Shape {
    static constexpr int kBox = 16;                                     // token rows of one TMA box
    static constexpr int kHalf = NT * 128;                              // bytes of one 64-wide half of the tokens
    static constexpr int kStage = kCodeBytes + 2 * kHalf;
    static constexpr int kStages = NT == 64 ? 4 : 5;
    static constexpr size_t kSmem = static_cast<size_t>(kStages) * kStage + 1024;  // + 8 (E + 1) bytes of tile table
};

// The group scales of one weight row: the thread of the row asks for those of its next tile a tile ahead (a load takes up to three
// groups under load), keeps them in registers until the tile is done and then leaves them in its own row of shared memory.
struct RowScales {
    uint4 ahead[2];
    const __half* row;
    uint32_t at;
    __device__ __forceinline__ void ask(const W8Shape& p, int e, int wrow) {
        row = p.scale + (static_cast<int64_t>(e) * p.N + min(wrow, p.N - 1)) * (p.K / p.group);
        if (p.scale_vecs > 0) ahead[0] = __ldg(reinterpret_cast<const uint4*>(row));
        if (p.scale_vecs > 1) ahead[1] = __ldg(reinterpret_cast<const uint4*>(row) + 1);
    }
    __device__ __forceinline__ void keep(const W8Shape& p) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            if (v < p.scale_vecs) {
                const uint32_t u[4] = {ahead[v].x, ahead[v].y, ahead[v].z, ahead[v].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + 16u * v + 4u * i), "r"(u[i]) : "memory");
            }
        }
    }
    // `mine`: the row this tile works on (the one asked for last belongs to the next tile)
    __device__ __forceinline__ __half get(const W8Shape& p, const __half* mine, int g) const {
        const int k = p.group == 128 ? g : (g << 7) / p.group;
        if (p.scale_vecs == 0) return __ldg(mine + k);
        unsigned short h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(at + 2u * k));
        return __ushort_as_half(h);
    }
};

template <int NT>
__device__ __forceinline__ Tile tile_at(int i, const int* first, const int* tok, const W8Shape& p) {
    Tile t = find_tile(i, first, tok, p.E, NT, 16);
    const int m = t.row0;
    t.row0 = p.gate_up ? m * 128 : m * kTileRows;
    t.row1 = p.gate_up ? p.N / 2 + m * 128 : m * kTileRows + 128;
    return t;
}

__device__ __forceinline__ float ld_peer(uint32_t addr, int rank) {
    uint32_t there;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(there) : "memory");
    return v;
}

// SPLIT (exact form, dense, fewer tiles than SMs): the blocks of a cluster take a part of the groups each, one tile per cluster; every
// block leaves its sums in its own shared memory and finishes a part of the tokens from those of all, in rank order.
template <int NT, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) w8_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                              const W8Shape p) {
    using S = Shape<NT>;
    constexpr int kStages = S::kStages;
    extern __shared__ uint8_t raw[];
    __shared__ __align__(8) uint64_t s_bar[2 * kStages + 9];
    __shared__ __align__(16) uint8_t s_scale[kTileRows * kScaleStride];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage0 = (smem_u32(raw) + 1023u) & ~1023u;
    int* s_first = reinterpret_cast<int*>(raw + (stage0 - smem_u32(raw)) + static_cast<size_t>(kStages) * S::kStage);
    int* s_tok = s_first + p.E + 1;
    const uint32_t bars = smem_u32(s_bar);
    auto full = [&](int s) { return bars + 8u * s; };
    auto done = [&](int s) { return bars + 8u * (kStages + s); };
    auto a_full = [&](int w, int b) { return bars + 8u * (2 * kStages + 2 * w + b); };
    auto d_free = [&](int b) { return bars + 8u * (2 * kStages + 4 + b); };
    const uint32_t ex = bars + 8u * (2 * kStages + 6);
    auto drained = [&](int w) { return ex + 8u + 8u * w; };

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(done(s), 2);  // the MMAs of both tiles
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(a_full(0, b), 4);
            mbar_init(a_full(1, b), 4);
            mbar_init(d_free(b), 8);
            mbar_init(drained(b), 1);
        }
        mbar_init(ex, 8);
        mbar_fence_init();
    }
    if (warp == 17) tmem_alloc(smem_u32(&s_tmem), 512);
    if (tid == 512) {
        tma_prefetch_map(&map_w);
        tma_prefetch_map(&map_x);
    }
    if (p.seg) pdl_wait();  // segments and tokens come from earlier kernels; without segments only the token loads wait
    pdl_trigger();
    const int mt = p.gate_up ? (p.N / 2 + 127) / 128 : (p.N + kTileRows - 1) / kTileRows;
    if (warp == 0) fill_tiles(p, NT, mt, s_first, s_tok, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int tiles = s_first[p.E], groups = p.K >> 7;
    volatile int* abort = &s_abort;
    // this block's tiles and, of each, its groups
    const int rank = SPLIT ? blockIdx.x % p.parts : 0, tile0 = SPLIT ? blockIdx.x / p.parts : blockIdx.x, stride = SPLIT ? tiles : gridDim.x;
    const int g0 = SPLIT ? rank * groups / p.parts : 0, g1 = SPLIT ? (rank + 1) * groups / p.parts : groups;
    auto tile = [&](int i) { return tile_at<NT>(i, s_first, s_tok, p); };

    if (warp >= 16) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == 16) {
        // ---- TMA: one thread ---------------------------------------------------------------------------------------
        if (elect_one()) {
            int s = 0, issued = 0, early = 0;
            uint32_t ph = 1;
            bool ok = true;
            Tile t = tile(tile0);
            auto stage_at = [&](int k) { return stage0 + static_cast<uint32_t>(k) * S::kStage; };
            auto bytes_of = [&](const Tile& x) { return kCodeBytes + 2u * ((x.n + S::kBox - 1) / S::kBox) * S::kBox * 128u; };
            auto load_codes = [&](const Tile& x, int g, int k) {
                mbar_expect_tx(full(k), bytes_of(x));
                tma_load_2d(stage_at(k), &map_w, g * 128, x.e * p.N + x.row0, full(k));
                tma_load_2d(stage_at(k) + kCodeBytes / 2, &map_w, g * 128, x.e * p.N + x.row1, full(k));
            };
            if (!p.seg) {  // the codes of the first stages do not depend on earlier kernels: on their way while those finish
                if (tile0 < tiles)
                    for (; early < min(kStages, g1 - g0); ++early) load_codes(t, g0 + early, early);
                pdl_wait();
            }
            for (int i = tile0; i < tiles && ok; i += stride) {
                Tile next = t;
                for (int g = g0; g < g1; ++g) {
                    if (issued >= early) {
                        if (!(ok = thread_wait(done(s), ph, abort))) break;
                        load_codes(t, g, s);
                    }
                    const uint32_t at = stage_at(s) + kCodeBytes;
                    for (int b = 0; b * S::kBox < t.n; ++b) {
                        tma_load_2d(at + b * S::kBox * 128, &map_x, g * 128, t.t0 + b * S::kBox, full(s));
                        tma_load_2d(at + S::kHalf + b * S::kBox * 128, &map_x, g * 128 + 64, t.t0 + b * S::kBox, full(s));
                    }
                    ++issued;
                    if (++s == kStages) { s = 0; ph ^= 1; }
                    if (g == g0) next = tile(i + stride);
                }
                t = next;
            }
            if (!ok) {  // gave up: the copies in flight still land in this block's shared memory
                for (int j = max(0, issued - kStages); j < issued; ++j) mbar_wait(full(j % kStages), (j / kStages) & 1);
            }
        }
    } else if (warp == 17 || warp == 18) {
        // ---- MMA: one thread per M tile ------------------------------------------------------------------------------
        if (elect_one()) {
            const int w = warp - 17;
            int s = 0, it = 0;
            bool ok = true;
            Tile t = tile(tile0);
            for (int i = tile0; i < tiles && ok; i += stride) {
                const uint32_t idesc = idesc_f16(128, max(16, (t.n + 15) & ~15), false);
                for (int g = g0; g < g1; ++g, ++it) {
                    const int b = it & 1;
                    // a widening warp has seen the stage's copies land before it arrives: no wait on full(s) here
                    if (!(ok = thread_wait(a_full(w, b), (it >> 1) & 1, abort))) break;
                    if (!(ok = thread_wait(d_free(b), ((it >> 1) & 1) ^ 1, abort))) break;
                    tc_fence_after();
                    const uint64_t x0 = smem_desc_sw128(stage0 + static_cast<uint32_t>(s) * S::kStage + kCodeBytes, 1024);
                    const uint32_t a = tmem + kColA + 128u * w + 64u * b, d = tmem + 128u * w + 64u * b;
#pragma unroll
                    for (int k = 0; k < 8; ++k) mma_f16_ts(d, a + 8u * k, x0 + (k >> 2) * (S::kHalf >> 4) + (k & 3) * 2u, idesc, k != 0);
                    // one event ends the group for everybody: the stage may be refilled, the A buffer rewritten, D read
                    tc_commit(done(s));
                    if (++s == kStages) s = 0;
                    if (g + 1 == g1) t = tile(i + stride);
                }
            }
            if (!ok) {  // gave up: nothing may still write TMEM when it is freed
                tc_commit(drained(w));
                mbar_wait(drained(w), 0);
            }
        }
    } else if (warp >= 8 && warp < 16) {
        // ---- widen: thread = weight row ----------------------------------------------------------------------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsWiden));
        const int w = (warp >> 2) & 1, row = tid & 127;
        const uint32_t to0 = tmem + (static_cast<uint32_t>(warp & 3) << 21) + kColA + 128u * w;
        const uint32_t from0 = stage0 + w * (kCodeBytes / 2) + row * 128u, swz = row & 7;
        int s = 0, it = 0, s2 = kStages - 2;       // s2, ph2: stage and phase of group it - 2, the last user of this A buffer
        uint32_t ph = 0, ph2 = 1;
        bool ok = true;
        for (int i = tile0; i < tiles && ok; i += stride) {
            for (int g = g0; g < g1; ++g, ++it) {
                const int b = it & 1;
                if (!(ok = warp_wait(full(s), ph, abort) && warp_wait(done(s2), ph2, abort))) break;
                tc_fence_after();
                const uint32_t from = from0 + static_cast<uint32_t>(s) * S::kStage, to = to0 + 64u * b;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    uint32_t a[16];
#pragma unroll
                    for (int c = 0; c < 2; ++c) widen16<false>(lds128(from + ((static_cast<uint32_t>(2 * h + c) ^ swz) << 4)), __half(), a + 8 * c);
                    tmem_st16(to + 16u * h, a);
                }
                tmem_wait_st();
                tc_fence_before();
                warp_arrive(a_full(w, b));
                if (++s == kStages) { s = 0; ph ^= 1; }
                if (++s2 == kStages) { s2 = 0; ph2 ^= 1; }
            }
        }
    } else if (warp < 8) {
        // ---- collect: thread = weight row --------------------------------------------------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCollect));
        pdl_wait();  // the residual is an earlier kernel's, and y may still be read by one
        const int w = warp >> 2, row = tid & 127;
        const uint32_t lanes = static_cast<uint32_t>(warp & 3) << 21;  // TMEM lane field
        const int half_rows = p.N / 2;
        int it = 0, round = 0, s = 0;
        uint32_t ph = 0;
        bool ok = true;
        Tile t = tile(tile0);
        RowScales sc;
        sc.at = smem_u32(s_scale) + (w * 128 + row) * kScaleStride;
        if (tile0 < tiles) sc.ask(p, t.e, (w ? t.row1 : t.row0) + row);
        for (int i = tile0; i < tiles && ok; i += stride, ++round) {
            const int lim = p.gate_up ? half_rows : p.N;                 // rows of this tile's kind
            const int mrow = (p.gate_up ? t.row0 : (w ? t.row1 : t.row0)) + row;  // gate/up: both tiles count gate rows
            const bool live = mrow < lim;
            Tile next = t;
            float acc[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) acc[j] = 0.f;
            const __half* mine = sc.row;
            sc.keep(p);
            for (int g = g0; g < g1; ++g, ++it) {
                const int db = it & 1;
                const float scale = __half2float(sc.get(p, mine, g));
                if (!(ok = warp_wait(done(s), ph, abort))) break;
                tc_fence_after();
                const uint32_t d = tmem + lanes + 128u * w + 64u * db;
#pragma unroll
                for (int c = 0; c < NT; c += 16) {
                    if (c < t.n) {
                        uint32_t r[16];
                        tmem_ld16(r, d + c);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(scale, __uint_as_float(r[j]), acc[c + j]);
                    }
                }
                tc_fence_before();
                // gate/up: the last sums' columns carry the exchange below and are freed after it
                if (!p.gate_up || g + 1 < g1) warp_arrive(d_free(db));
                if (++s == kStages) { s = 0; ph ^= 1; }
                if (g == g0) {
                    next = tile(i + stride);
                    if (i + stride < tiles) sc.ask(p, next.e, (w ? next.row1 : next.row0) + row);
                }
            }
            if (!ok) break;
            const int dl = (it - 1) & 1;  // buffer of the last group

            if (SPLIT) {
                // every group of this block has been read: the stages are free for its sums, [token][row]
                const uint32_t at = stage0 + 4u * (w * 128 + row);
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    if (j < t.n) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4u * kTileRows * j), "f"(acc[j]) : "memory");
            } else if (p.gate_up) {
                // SwiGLU: the gate tile's threads finish the first half of the tokens, the up tile's the second; what the other
                // needs goes through the accumulators' own columns of TMEM (same lanes, so no shared memory)
                constexpr int H = NT / 2;
                uint32_t r[16];
#pragma unroll
                for (int c = 0; c < H; c += 16) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = c + j < H ? __float_as_uint(w ? acc[c + j < H ? c + j : 0] : acc[H + (c + j < H ? c + j : 0)]) : 0u;
                    tmem_st16(tmem + lanes + 128u * w + 64u * dl + c, r);
                }
                tmem_wait_st();
                tc_fence_before();
                warp_arrive(ex);
                if (!(ok = warp_wait(ex, round & 1, abort))) break;
                tc_fence_after();
                const uint32_t d_other = tmem + lanes + 128u * (w ^ 1) + 64u * dl;
                const int first = w ? H : 0;
#pragma unroll
                for (int c = 0; c < H; c += 16) {
                    if (first + c < t.n) {
                        tmem_ld16(r, d_other + c);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16 && c + j < H; j += 2) {
                            float y[2];
                            const float o0 = __uint_as_float(r[j]), o1 = __uint_as_float(r[j + 1]);
                            if (w) swiglu2(o0, acc[H + c + j], o1, acc[H + c + j + 1], y[0], y[1]);
                            else swiglu2(acc[c + j], o0, acc[c + j + 1], o1, y[0], y[1]);
#pragma unroll
                            for (int v = 0; v < 2; ++v)
                                if (live && first + c + j + v < t.n)
                                    p.y[static_cast<int64_t>(t.t0 + first + c + j + v) * half_rows + mrow] = __float2half_rn(y[v]);
                        }
                    }
                }
                tc_fence_before();
                warp_arrive(d_free(dl));
            } else if (live) {
                __half* y = p.y + static_cast<int64_t>(t.t0) * p.N + mrow;
                float* y32 = p.y32 + static_cast<int64_t>(t.t0) * p.N + mrow;
                const __half* res = p.resid ? p.resid + static_cast<int64_t>(t.t0) * p.N + mrow : nullptr;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    if (j < t.n) {
                        if (p.y32) {
                            y32[static_cast<int64_t>(j) * p.N] = acc[j];
                            continue;
                        }
                        __half v = __float2half_rn(acc[j]);
                        if (res) v = __hadd(v, res[static_cast<int64_t>(j) * p.N]);
                        y[static_cast<int64_t>(j) * p.N] = v;
                    }
                }
            }
            t = next;
        }
    }
    if (SPLIT) {
        __syncwarp();
        cluster_sync();
        const Tile t = tile(tile0);
        const int mrow = t.row0 + tid;  // row1 follows row0 (dense)
        if (warp < 8 && mrow < p.N) {
            const int per = (t.n + p.parts - 1) / p.parts, j1 = min(t.n, (rank + 1) * per);
            for (int j = rank * per; j < j1; ++j) {
                float part[8], sum = 0.f;
#pragma unroll
                for (int r = 0; r < 8; ++r) part[r] = r < p.parts ? ld_peer(stage0 + 4u * (kTileRows * j + tid), r) : 0.f;
#pragma unroll
                for (int r = 0; r < 8; ++r) sum += part[r];
                const int64_t o = static_cast<int64_t>(t.t0 + j) * p.N + mrow;
                __half v = __float2half_rn(sum);
                if (p.resid) v = __hadd(v, p.resid[o]);
                p.y[o] = v;
            }
        }
        cluster_sync();  // nobody leaves while its sums are read
    }
    __syncthreads();
    if (tid == 0 && s_abort && p.err_flag) atomicOr(p.err_flag, LEMOQ_FLAG_WAIT_TIMEOUT);
    if (warp == 17) {
        tc_fence_after();
        tmem_free(tmem, 512);
    }
}

template <int NT>
int launch_nt(W8Shape p, const __half* x, const int8_t* codes, const LaunchCfg& lc) {
    CUtensorMap map_w, map_x;
    if (int rc = encode_rows_map(&map_w, codes, 1, static_cast<int64_t>(p.E) * p.N, p.K, 128)) return rc;
    if (int rc = encode_rows_map(&map_x, x, 2, p.T, p.K, Shape<NT>::kBox)) return rc;
    const size_t smem = Shape<NT>::kSmem + 8 * (static_cast<size_t>(p.E) + 1);
    const int gk = p.K / p.group;
    p.scale_vecs = aligned16(p.scale) && (gk == 8 || gk == 16) ? gk / 8 : 0;
    const int64_t mt = p.gate_up ? (p.N / 2 + 127) / 128 : (p.N + kTileRows - 1) / kTileRows;
    const int64_t most = mt * (p.seg ? p.T / NT + std::min<int64_t>(p.E, p.T) : (p.T + NT - 1) / NT);  // tiles, at most
    const int sms = sm_count();
    // A linear of few rows is a tile on every sixth SM or fewer (2048 rows: 8 tiles), each a chain of K / 128 groups of half a
    // microsecond: its groups are shared out over a cluster while that leaves every block two of them and an SM of its own.
    int parts = 1;
    while (parts < 8 && most * 2 * parts <= sms && 4 * parts <= p.K >> 7) parts *= 2;
    if (parts > 1 && !p.seg && !p.gate_up && !p.y32 && p.T <= NT) {
        if (int rc = allow_smem(w8_gemm_kernel<NT, true>, smem)) return rc;
        p.parts = parts;
        LaunchCfg clustered = lc;
        clustered.cluster = parts;
        return launch_kernel(w8_gemm_kernel<NT, true>, dim3(static_cast<unsigned>(most) * parts), dim3(kThreads), smem, clustered, map_w, map_x, p);
    }
    if (int rc = allow_smem(w8_gemm_kernel<NT, false>, smem)) return rc;
    const int grid = static_cast<int>(std::min<int64_t>(sms, std::max<int64_t>(most, 1)));
    return launch_kernel(w8_gemm_kernel<NT, false>, dim3(grid), dim3(kThreads), smem, lc, map_w, map_x, p);
}

}  // namespace

int launch_w8_gemm(const W8GemmParams& g, const LaunchCfg& lc) {
    W8Shape p = {};
    p.T = g.T; p.N = g.N; p.K = g.K; p.group = g.group_size; p.E = g.E; p.gate_up = g.gate_up ? 1 : 0;
    p.seg = g.seg; p.scale = g.scale; p.resid = g.resid; p.y = g.y; p.y32 = g.y32; p.err_flag = g.err_flag;
    // NT bounds the tokens of a tile, the MMA's N follows the real count: a small NT only saves registers and stage bytes, a
    // large one saves widening the same codes again for a second token tile.  Twice the mean per expert covers nearly all.
    const int64_t want = g.seg ? 2 * ((static_cast<int64_t>(g.T) + g.E - 1) / g.E) : g.T;
    if (want <= 16) return launch_nt<16>(p, g.x, g.codes, lc);
    if (want <= 32) return launch_nt<32>(p, g.x, g.codes, lc);
    if (want <= kExactTokens || g.exact) return launch_nt<kExactTokens>(p, g.x, g.codes, lc);
    return launch_w8_pair(p, g.x, g.codes, lc);
}

}  // namespace lemoq

using namespace lemoq;

extern "C" int lemoq_w8_gemm(const void* x, int T, const int8_t* codes, const void* scale, int N, int K, int group_size, const int32_t* seg_offsets,
                             int E, int gate_up, int exact, const void* resid, void* y, int* err_flag, void* stream) {
    LEMOQ_REQUIRE(T >= 0 && N > 0 && K > 0 && E >= 1, LEMOQ_ERR_INVALID, "w8_gemm: bad shape");
    LEMOQ_REQUIRE(!gate_up || N % 2 == 0, LEMOQ_ERR_UNSUPPORTED, "w8_gemm: gate/up needs an even number of rows");
    LEMOQ_REQUIRE(K % 128 == 0, LEMOQ_ERR_UNSUPPORTED, "w8_gemm: K=%d must be a multiple of 128", K);
    LEMOQ_REQUIRE(group_size > 0 && K % group_size == 0, LEMOQ_ERR_INVALID, "w8_gemm: bad group_size %d", group_size);
    LEMOQ_REQUIRE(group_size % 128 == 0, LEMOQ_ERR_UNSUPPORTED, "w8_gemm: group_size=%d must be a multiple of 128", group_size);
    LEMOQ_REQUIRE(E == 1 || seg_offsets, LEMOQ_ERR_INVALID, "w8_gemm: several experts need segment offsets");
    LEMOQ_REQUIRE(E <= kMaxExperts, LEMOQ_ERR_UNSUPPORTED, "w8_gemm: E=%d above %d", E, kMaxExperts);
    LEMOQ_REQUIRE(!(gate_up && resid), LEMOQ_ERR_UNSUPPORTED, "w8_gemm: no residual in gate/up mode");
    LEMOQ_REQUIRE(static_cast<int64_t>(E) * N <= 0x7fffffff, LEMOQ_ERR_UNSUPPORTED, "w8_gemm: too many rows");
    if (T == 0) return LEMOQ_OK;
    LEMOQ_REQUIRE(x && codes && scale && y && aligned16(x) && aligned16(codes), LEMOQ_ERR_INVALID, "w8_gemm: null or unaligned pointer");
    W8GemmParams g;
    g.x = reinterpret_cast<const __half*>(x);
    g.codes = codes;
    g.scale = reinterpret_cast<const __half*>(scale);
    g.seg = seg_offsets;
    g.resid = reinterpret_cast<const __half*>(resid);
    g.y = reinterpret_cast<__half*>(y);
    g.T = T; g.N = N; g.K = K; g.group_size = group_size; g.E = E; g.gate_up = gate_up != 0;
    g.exact = exact != 0;
    g.err_flag = err_flag ? err_flag : status_word();
    LaunchCfg lc;
    lc.stream = static_cast<cudaStream_t>(stream);
    return launch_w8_gemm(g, lc);
}
