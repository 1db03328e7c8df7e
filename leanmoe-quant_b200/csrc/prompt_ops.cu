// Row operations between the tensor-core kernels when many tokens go through a layer at once.  All of them are bounded by
// the rows they read and write (L2-resident up to some thousand tokens); each does everything that touches its rows in one
// pass, so that a layer is nine launches (four of them GEMMs, one attention):
//
//   embed_norm     embedding row, input RMSNorm                                   one block per token
//   qkv_rows       q/k RMSNorm over the projection width, RoPE, rows into the caches one block per token
//   norm_route     post-attention RMSNorm, router logits (fp16 mma), softmax, top-k  one block per 16 tokens
//   place_rows     activations into expert order, from norm_route's counts           one block per 1 to 16 tokens
//   pair_plan      the same where only expert ids are given, or of very many tokens: stable counting sort, one block per expert
//   gather_rows    and the copy (few pairs: done by pair_plan)                       one block per pair
//   combine_norm   routing-weighted sum in slot order (fp32) + residual, next norm   one block per token
#include "prompt.h"
#include "stream.cuh"

#include <algorithm>
#include <type_traits>

namespace lemoq {
namespace {

constexpr int kRowThreads = 256;
constexpr int kRowVecs = 2;  // 8-value vectors a thread keeps: rows up to 4096

// RMSNorm of a row held as fp32 in registers (vector v at 8 * (tid + 256 v)); HF rounding chain, fp16 out.
__device__ __forceinline__ void norm_row_store(const float (&f)[kRowVecs][8], int H, const __half* __restrict__ w, float eps, __half* __restrict__ y, float* red) {
    uint4 wv[kRowVecs];  // on their way under the reduction
#pragma unroll
    for (int v = 0; v < kRowVecs; ++v)
        if (8 * (threadIdx.x + kRowThreads * v) < H) wv[v] = __ldg(reinterpret_cast<const uint4*>(w + 8 * (threadIdx.x + kRowThreads * v)));
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < kRowVecs; ++v)
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(f[v][j], f[v][j], ss);  // vectors beyond the row are zero
    ss = block_sum(ss, red);
    const float rstd = 1.0f / sqrtf(ss / static_cast<float>(H) + eps);
#pragma unroll
    for (int v = 0; v < kRowVecs; ++v) {
        const int i = 8 * (threadIdx.x + kRowThreads * v);
        if (i < H) {
            const __half* wh = reinterpret_cast<const __half*>(&wv[v]);
            __align__(16) __half o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = __hmul(__float2half_rn(f[v][j] * rstd), wh[j]);
            *reinterpret_cast<uint4*>(y + i) = *reinterpret_cast<const uint4*>(o);
        }
    }
}

__global__ void __launch_bounds__(kRowThreads) embed_norm_kernel(const int64_t* __restrict__ tokens, const __half* __restrict__ embed, int64_t vocab, int H,
                                                                 const __half* __restrict__ w, float eps, __half* __restrict__ x, __half* __restrict__ h, int* err) {
    __shared__ float red[40];
    pdl_wait();
    pdl_trigger();
    const int64_t t = blockIdx.x, tok = checked_token(tokens + t, vocab, err);
    float f[kRowVecs][8];
#pragma unroll
    for (int v = 0; v < kRowVecs; ++v) {
        const int i = 8 * (threadIdx.x + kRowThreads * v);
        uint4 e = make_uint4(0, 0, 0, 0);
        if (i < H) {
            e = ld_stream16(embed + tok * H + i);
            *reinterpret_cast<uint4*>(x + t * H + i) = e;
        }
        unpack8_h(e, f[v]);
    }
    norm_row_store(f, H, w, eps, h + t * H, red);
}

// out[t] = fp16(sum_k w[t, k] * y[place[t, k]]) + x1[t]; then the next RMSNorm of it.  Bounded by the K rows a token reads: eight of them are in
// flight at a time, the residual and the norm weights beside them.  (Four at a time, the residual first and the norm weights
// last: 5.9 us alone at 61 tokens, now 4.6; the same 40 us at 4096, 4.6 TB/s.)
template <int VECS>  // vectors of eight values a thread has of a row
__global__ void __launch_bounds__(kRowThreads) combine_norm_kernel(const __half* __restrict__ y, const int32_t* __restrict__ place, const float* __restrict__ top_w,
                                                                   int K, const __half* __restrict__ x1, int H, const __half* __restrict__ w, float eps,
                                                                   __half* __restrict__ x2, __half* __restrict__ h) {
    __shared__ float red[40];
    pdl_wait();
    pdl_trigger();
    const int64_t t = blockIdx.x;
    float f[kRowVecs][8];
    uint4 r[VECS];
#pragma unroll
    for (int v = 0; v < kRowVecs; ++v)
#pragma unroll
        for (int j = 0; j < 8; ++j) f[v][j] = 0.f;
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        const int i = 8 * (threadIdx.x + kRowThreads * v);
        if (i < H) r[v] = ld_cg16(x1 + t * H + i);
    }
    for (int k0 = 0; k0 < K; k0 += 8) {
        uint4 e[VECS][8];
        float wk[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k0 + k < K) {
                wk[k] = __half2float(__float2half_rn(__ldg(top_w + t * K + k0 + k)));
                const __half* src = y + static_cast<int64_t>(__ldg(place + t * K + k0 + k)) * H;
#pragma unroll
                for (int v = 0; v < VECS; ++v) {
                    const int i = 8 * (threadIdx.x + kRowThreads * v);
                    if (i < H) e[v][k] = ld_cg16(src + i);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k0 + k < K) {
#pragma unroll
                for (int v = 0; v < VECS; ++v) {
                    if (8 * (threadIdx.x + kRowThreads * v) < H) {
                        float g[8];
                        unpack8_h(e[v][k], g);
#pragma unroll
                        for (int j = 0; j < 8; ++j) f[v][j] = __fadd_rn(f[v][j], __fmul_rn(g[j], wk[k]));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        const int i = 8 * (threadIdx.x + kRowThreads * v);
        if (i < H) {
            __half* rh = reinterpret_cast<__half*>(&r[v]);
#pragma unroll
            for (int j = 0; j < 8; ++j) rh[j] = __hadd(__float2half_rn(f[v][j]), rh[j]);
            *reinterpret_cast<uint4*>(x2 + t * H + i) = r[v];
            unpack8_h(r[v], f[v]);
        }
    }
    norm_row_store(f, H, w, eps, h + t * H, red);
}

// Per-token symmetric int8 of a head's 128 values, eight in each of 16 neighbouring lanes (fp32 amax, true division, half to even; the
// scale is stored as fp16).
__device__ __forceinline__ void quantise_head_store(const __half* x, int8_t* codes, __half* scale, bool first_lane) {
    float f[8], amax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        f[j] = __half2float(x[j]);
        amax = fmaxf(amax, fabsf(f[j]));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(threadIdx.x & 16 ? 0xffff0000u : 0x0000ffffu, amax, o, 16));
    const float s = amax > 0.f ? __fdiv_rn(amax, 127.0f) : 1.0f;
    __align__(8) int8_t c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) c[j] = static_cast<int8_t>(static_cast<int>(fminf(fmaxf(rintf(__fdiv_rn(f[j], s)), -127.0f), 127.0f)));
    *reinterpret_cast<uint2*>(codes) = *reinterpret_cast<const uint2*>(c);
    if (first_lane) *scale = __float2half_rn(s);
}

// Sums over the block of two values per thread at once.
__device__ __forceinline__ float2 block_sum2(float2 v, float2* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float2 t = lane < kRowThreads / 32 ? red[lane] : make_float2(0.f, 0.f);
    t.x = warp_sum(t.x);
    t.y = warp_sum(t.y);
    return t;
}

// One block per token, A = heads * 128 <= 4096.  qkv (T, 3A) -> q (T, A) normalised and rotated.  The k and v rows go into slot pos[t] of
// the fp16 caches (heads, S, 128), or (INT8, lockstep decoding) quantised into slot *pos of the row's own caches (T * heads, S, 128).
// Bounded by the rows read and written; everything a thread needs is asked for at once.  (v rows, norm weights and angles where they were used,
// a reduction for q and one for k: 5.5, 10.5 and 33.5 us alone at 61, 1024 and 4096 tokens; now 3.6, 7.5 and 22.)
template <bool INT8, int VECS>  // vectors of eight values a thread has of a row
__global__ void __launch_bounds__(kRowThreads) qkv_rows_kernel(const QkvRows p) {
    __shared__ float2 red[kRowThreads / 32];
    __shared__ __align__(16) __half row[2][kRowThreads * 8 * VECS];
    const int64_t t = blockIdx.x;
    const int A = p.heads * 128, tid = threadIdx.x;
    uint4 w[2][VECS];  // norm weights: not an earlier kernel's
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        const int i = 8 * (tid + kRowThreads * v);
        if (i < A) {
            w[0][v] = __ldg(reinterpret_cast<const uint4*>(p.q_norm + i));
            w[1][v] = __ldg(reinterpret_cast<const uint4*>(p.k_norm + i));
        }
    }
    pdl_wait();
    pdl_trigger();
    const __half* src = p.qkv + t * 3 * A;
    uint4 x[3][VECS];
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        const int i = 8 * (tid + kRowThreads * v);
#pragma unroll
        for (int m = 0; m < 3; ++m) x[m][v] = i < A ? ld_cg16(src + m * A + i) : make_uint4(0, 0, 0, 0);
    }
    int64_t pos = p.pos[INT8 ? 0 : t];
    if (pos < 0 || pos >= p.S) {
        if (p.err_flag && tid == 0) atomicOr(p.err_flag, LEMOQ_FLAG_BAD_POSITION);
        pos = pos < 0 ? 0 : p.S - 1;
    }
    const int d = 8 * tid & 127;  // the same in every vector of a thread
    const uint4 cos = __ldg(reinterpret_cast<const uint4*>(p.rope_cos + pos * 128 + d)), sin = __ldg(reinterpret_cast<const uint4*>(p.rope_sin + pos * 128 + d));
    float2 ss = make_float2(0.f, 0.f);
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        float f[8];
        unpack8_h(x[0][v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss.x = fmaf(f[j], f[j], ss.x);
        unpack8_h(x[1][v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss.y = fmaf(f[j], f[j], ss.y);
    }
    ss = block_sum2(ss, red);
    const float rstd[2] = {1.0f / sqrtf(ss.x / static_cast<float>(A) + p.eps), 1.0f / sqrtf(ss.y / static_cast<float>(A) + p.eps)};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int v = 0; v < VECS; ++v) {
            const int i = 8 * (tid + kRowThreads * v);
            if (i < A) {
                const __half* wh = reinterpret_cast<const __half*>(&w[m][v]);
                float f[8];
                unpack8_h(x[m][v], f);
                __align__(16) __half o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = __hmul(__float2half_rn(f[j] * rstd[m]), wh[j]);
                x[m][v] = *reinterpret_cast<const uint4*>(o);
                *reinterpret_cast<uint4*>(&row[m][i]) = x[m][v];
            }
        }
    }
    __syncwarp();  // the other half of a head is eight lanes away
    float c[8], s[8];
    unpack8_h(cos, c);
    unpack8_h(sin, s);
    const int away = d < 64 ? 64 : -64;
    const float sign = d < 64 ? -1.f : 1.f;
#pragma unroll
    for (int v = 0; v < VECS; ++v) {
        const int i = 8 * (tid + kRowThreads * v);
        if (i < A) {
            const int64_t row_at = (INT8 ? t * p.heads + (i >> 7) : static_cast<int64_t>(i >> 7)) * p.S + pos, slot = row_at * 128 + d;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                float a[8], b[8];
                unpack8_h(x[m][v], a);
                unpack8_h(*reinterpret_cast<const uint4*>(&row[m][i + away]), b);
                __align__(16) __half o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = __float2half_rn(__fadd_rn(__fmul_rn(a[j], c[j]), __fmul_rn(sign * b[j], s[j])));
                if (INT8 && m) {
                    quantise_head_store(o, p.kc + slot, p.ks + row_at, d == 0);
                } else {
                    __half* dst = m ? p.keys + slot : p.q + t * A + i;
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
                }
            }
            if (INT8)
                quantise_head_store(reinterpret_cast<const __half*>(&x[2][v]), p.vc + slot, p.vs + row_at, d == 0);
            else
                *reinterpret_cast<uint4*>(p.values + slot) = x[2][v];
        }
    }
}

// ---- router ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int kRouteWarps = 16;
constexpr int kRouteTokens = 16;

// A warp normalises one of the block's 16 rows; then the warps split H for the logits of all 16 rows and all experts.  Their partial
// sums meet in shared memory (over the rows) and are added in warp order.  With 0.27 GFLOP per thousand tokens the work is too small for
// a tcgen05 pipeline to fill: what counts is one round of loads, so a row and its norm weights are asked for together, and a warp's first router
// values before the previous kernel ends (the rest of the router is asked into L2).  A and B use the same permutation of k inside 32
// values, so that 128-bit loads feed the fragments.  The top-k takes the bits of a probability as a whole number: two warp-wide reductions a choice.
// (As a norm kernel and a router kernel of eight warps with all loads in turn: 3.5 + 19 us at 64 tokens; with loads inside loops and a choice by
// ten shuffles a layer of a prompt of 61 tokens took 2.8 us more than with this, of a step of 11 sequences 5.6, of one of 64 at 2048 3.)
template <int TILES, int VECS>  // expert tiles of 8; vectors of eight values a lane has of a row
__global__ void __launch_bounds__(kRouteWarps * 32) norm_route_kernel(const __half* __restrict__ x, const __half* __restrict__ norm_w, float eps,
                                                                      const __half* __restrict__ router, int T, int H, int E, int top_k, int norm,
                                                                      __half* __restrict__ h, float* __restrict__ top_w, int32_t* __restrict__ top_i, int32_t* __restrict__ rank,
                                                                      int32_t* __restrict__ counts) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ int s_ids[kRouteTokens * 32];  // expert of the block's pairs, -1 behind the end
    float* part = reinterpret_cast<float*>(smem);    // [warp][16 tokens][E], after the rows
    __half* rows = reinterpret_cast<__half*>(smem);  // [16][H + 8]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int t0 = blockIdx.x * kRouteTokens, tiles = E >> 3, pitch = H + 8;
    for (int i = (blockIdx.x % 4) * kRouteWarps * 32 + threadIdx.x; i < E * H / 64; i += 4 * kRouteWarps * 32)  // four blocks share it
        asm volatile("prefetch.global.L2 [%0];" ::"l"(router + 64 * static_cast<int64_t>(i)));
    const __half* wr = router + static_cast<int64_t>(g) * H + 8 * q;
    constexpr bool kAhead = TILES <= 8, kNormAhead = VECS <= 8;  // (where the registers are there for it)
    uint4 w[8];
    auto load_router = [&](int k, int n0) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
            if (n0 + n < tiles) w[n] = __ldg(reinterpret_cast<const uint4*>(wr + static_cast<int64_t>(8 * (n0 + n)) * H + k));
    };
    if (kAhead && 32 * warp < H) load_router(32 * warp, 0);
    uint4 wv[VECS];
#pragma unroll
    for (int v = 0; v < VECS; ++v)
        if (kNormAhead && 8 * lane + 256 * v < H) wv[v] = __ldg(reinterpret_cast<const uint4*>(norm_w + 8 * lane + 256 * v));
    pdl_wait();
    pdl_trigger();
    {
        const int t = t0 + warp;
        __half* mine = rows + warp * pitch;
        if (t < T) {
            const __half* src = x + static_cast<int64_t>(t) * H;
            uint4 r[VECS];
#pragma unroll
            for (int v = 0; v < VECS; ++v) r[v] = 8 * lane + 256 * v < H ? ld_cg16(src + 8 * lane + 256 * v) : make_uint4(0, 0, 0, 0);
            float ss = 0.f;
#pragma unroll
            for (int v = 0; v < VECS; ++v) {
                float f[8];
                unpack8_h(r[v], f);
#pragma unroll
                for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);  // vectors behind the row are zero
            }
            const float rstd = 1.0f / sqrtf(warp_sum(ss) / static_cast<float>(H) + eps);
#pragma unroll
            for (int v = 0; v < VECS; ++v) {
                const int i = 8 * lane + 256 * v;
                if (i < H) {
                    if (!kNormAhead) wv[v] = __ldg(reinterpret_cast<const uint4*>(norm_w + i));
                    const __half *vh = reinterpret_cast<const __half*>(&r[v]), *wh = reinterpret_cast<const __half*>(&wv[v]);
                    __align__(16) __half o[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = __hmul(__float2half_rn(__half2float(vh[j]) * rstd), wh[j]);
                    *reinterpret_cast<uint4*>(mine + i) = *reinterpret_cast<const uint4*>(o);
                    *reinterpret_cast<uint4*>(h + static_cast<int64_t>(t) * H + i) = *reinterpret_cast<const uint4*>(o);
                }
            }
        } else {
            for (int i = 8 * lane; i < H; i += 256) *reinterpret_cast<uint4*>(mine + i) = make_uint4(0, 0, 0, 0);
        }
    }
    __syncthreads();
    float c[TILES][4];
#pragma unroll
    for (int n = 0; n < TILES; ++n) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
    for (int k = 32 * warp; k < H; k += 32 * kRouteWarps) {
        const uint4 a = *reinterpret_cast<const uint4*>(rows + g * pitch + 8 * q + k), b = *reinterpret_cast<const uint4*>(rows + (g + 8) * pitch + 8 * q + k);
#pragma unroll
        for (int n0 = 0; n0 < TILES; n0 += 8) {
            if (!kAhead) load_router(k, n0);
            uint4 u[8];
#pragma unroll
            for (int n = 0; n < 8; ++n) u[n] = w[n];
            if (kAhead && k + 32 * kRouteWarps < H) load_router(k + 32 * kRouteWarps, 0);  // on its way under the work on this
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                if (n0 + n < tiles) {
                    mma_f16(c[n0 + n], a.x, b.x, a.y, b.y, u[n].x, u[n].y);
                    mma_f16(c[n0 + n], a.z, b.z, a.w, b.w, u[n].z, u[n].w);
                }
            }
        }
    }
    __syncthreads();
    float* mine = part + warp * kRouteTokens * E;
#pragma unroll
    for (int n = 0; n < TILES; ++n) {
        if (n < tiles) {
            *reinterpret_cast<float2*>(mine + g * E + 8 * n + 2 * q) = make_float2(c[n][0], c[n][1]);
            *reinterpret_cast<float2*>(mine + (g + 8) * E + 8 * n + 2 * q) = make_float2(c[n][2], c[n][3]);
        }
    }
    __syncthreads();
    constexpr int PER = TILES / 4 < 1 ? 1 : TILES / 4;  // experts of a lane: lane + 32 i
    const int t = t0 + warp;
    static_assert(kRouteTokens == kRouteWarps, "a warp chooses for one token");
    if (lane < top_k) s_ids[warp * top_k + lane] = -1;
    if (t < T) {
        float p[PER];
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = lane + 32 * i;
            p[i] = -INFINITY;
            if (e < E) {
                float v = 0.f;
#pragma unroll
                for (int u = 0; u < kRouteWarps; ++u) v += part[(u * kRouteTokens + warp) * E + e];
                p[i] = __half2float(__float2half_rn(v));  // the logits are fp16 values
            }
            mx = fmaxf(mx, p[i]);
        }
        mx = warp_max(mx);
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (lane + 32 * i < E) {
                p[i] = expf(p[i] - mx);
                sum += p[i];
            }
        }
        sum = warp_sum(sum);
        int key[PER];  // order of the probabilities; -1 taken or no expert.  If one is not a number, none is: the first experts, and weights that are none either
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const float v = p[i] / sum;
            key[i] = lane + 32 * i < E ? (v >= 0.f ? __float_as_int(v) : 0x7fffffff) : -1;
        }
        float kept = 0.f, wsum = 0.f;
        int kept_i = 0;
        for (int k = 0; k < top_k; ++k) {
            int top = key[0];
#pragma unroll
            for (int i = 1; i < PER; ++i) top = max(top, key[i]);
            top = __reduce_max_sync(0xffffffffu, top);
            unsigned first = 0x7fffffffu;  // the lowest expert that has it
#pragma unroll
            for (int i = PER - 1; i >= 0; --i)
                if (key[i] == top) first = lane + 32 * i;
            const int bi = static_cast<int>(__reduce_min_sync(0xffffffffu, first));  // (there is one: top_k <= E)
            const float best = __int_as_float(top);
            wsum += best;
            if (lane == k) {
                kept = best;
                kept_i = bi;
            }
#pragma unroll
            for (int i = 0; i < PER; ++i)
                if (bi == lane + 32 * i) key[i] = -1;
        }
        if (lane < top_k) {
            top_w[static_cast<int64_t>(t) * top_k + lane] = norm ? kept / wsum : kept;
            top_i[static_cast<int64_t>(t) * top_k + lane] = kept_i;
            s_ids[warp * top_k + lane] = kept_i;
        }
    }
    // A warp's experts: how many of the block's pairs go to each, and which of them a pair is (in pair order).
    __syncthreads();
    for (int e = warp; e < E; e += kRouteWarps) {
        int n = 0;
        for (int i0 = 0; i0 < kRouteTokens * top_k; i0 += 32) {
            const int i = i0 + lane;
            const bool hit = i < kRouteTokens * top_k && s_ids[i] == e;
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) rank[static_cast<int64_t>(t0) * top_k + i] = n + __popc(m & ((1u << lane) - 1u));
            n += __popc(m);
        }
        if (lane == 0) counts[blockIdx.x * E + e] = n;
    }
}

// ---- pairs into expert order ----------------------------------------------------------------------------------------------
constexpr int kPlanThreads = 512;

template <typename ID>
__device__ __forceinline__ int expert_of(const ID* __restrict__ ids, int p, int E, int* err) {
    const ID e = ids[p];
    if (e >= 0 && e < E) return static_cast<int>(e);
    if (err) atomicOr(err, LEMOQ_FLAG_BAD_EXPERT);
    return e < 0 ? 0 : E - 1;
}

// One block per expert: counts the pairs of lower experts, then gives its own pairs their rows in pair order.  GATHER: it also copies
// the activations of its pairs, up to kGatherPairs of them in all: a launch less, but an expert with many pairs is one block's work.
// Us of a call of the experts' block (64 experts, 8 a token) with the gather in here / in a kernel of its own: 16 pairs 32.4 / 33.0, 32 49.4 / 50.5,
// 64 66.5 / 67.7, 128 77.3 / 78.0, 256 to 1024 the same within what two runs of one side differ by.  The pairs of very many tokens of a prompt,
// which are plain int32 ids, are always above the line.
constexpr int kGatherPairs = 1024;
template <typename ID, bool GATHER>
__global__ void __launch_bounds__(kPlanThreads) pair_plan_kernel(const ID* __restrict__ top_i, int P, int E, int32_t* __restrict__ place,
                                                                 int32_t* __restrict__ pair_of, int32_t* __restrict__ seg, const __half* __restrict__ h, int K, int H,
                                                                 __half* __restrict__ x_sorted, int* err) {
    __shared__ int s_warp[kPlanThreads / 32 + 1];
    __shared__ int s_mine[GATHER ? kGatherPairs : 1];
    const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    pdl_trigger();
    int below = 0;
    for (int p = threadIdx.x; p < P; p += kPlanThreads) below += expert_of(top_i, p, E, e == 0 ? err : nullptr) < e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    if (lane == 0) s_warp[warp] = below;
    __syncthreads();
    int base = 0;
#pragma unroll
    for (int w = 0; w < kPlanThreads / 32; ++w) base += s_warp[w];
    __syncthreads();
    if (threadIdx.x == 0) seg[e] = base;
    const int row0 = base;
    for (int p0 = 0; p0 < P; p0 += kPlanThreads) {
        const int p = p0 + threadIdx.x;
        const bool hit = p < P && expert_of<ID>(top_i, p, E, nullptr) == e;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kPlanThreads / 32; ++w) {
            const int n = s_warp[w];
            before += w < warp ? n : 0;
            all += n;
        }
        if (hit) {
            const int row = base + before + __popc(m & ((1u << lane) - 1u));
            place[p] = row;
            pair_of[row] = p;
            if (GATHER) s_mine[row - row0] = p;
        }
        base += all;
        __syncthreads();
    }
    if (e == E - 1 && threadIdx.x == 0) seg[E] = base;
    if (GATHER) {
        const int vecs = H / 8;
        const int total = (base - row0) * vecs;
        for (int u0 = threadIdx.x; u0 < total; u0 += 4 * kPlanThreads) {  // four loads in flight
            uint4 v[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int u = u0 + b * kPlanThreads, r = u / vecs;
                if (u < total) v[b] = ld_cg16(h + static_cast<int64_t>(s_mine[r] / K) * H + 8 * (u - r * vecs));
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int u = u0 + b * kPlanThreads, r = u / vecs;
                if (u < total) *reinterpret_cast<uint4*>(x_sorted + static_cast<int64_t>(row0 + r) * H + 8 * (u - r * vecs)) = v[b];
            }
        }
    }
}

// Rows into expert order after norm_route, whose blocks left the pairs of every expert among their 16 tokens (`counts`) and the place of a
// pair among those (`rank`): a block sums the counts of all blocks and of those before its tokens', which gives the first row of every
// expert and of its own tokens in it, and writes each of its rows `K` times.  Bounded by those writes.  Us of this kernel / of a counting sort
// by a block per expert and a gather by a block per pair, alone: 5.3 / 5.5 at 61 tokens, 12 / 23 at 1024, 39 / 77 at 4096.
constexpr int kPlaceThreads = 256;
__global__ void __launch_bounds__(kPlaceThreads) place_rows_kernel(const int32_t* __restrict__ top_i, const int32_t* __restrict__ rank, const int32_t* __restrict__ counts,
                                                                   int T, int K, int E, const __half* __restrict__ h, int H, int per_block, int32_t* __restrict__ place,
                                                                   int32_t* __restrict__ seg, __half* __restrict__ x_sorted) {
    __shared__ int s_all[kPlaceThreads], s_below[kPlaceThreads], s_base[128], s_row[kRouteTokens * 32];
    const int tid = threadIdx.x, t0 = blockIdx.x * per_block, chunks = (T + kRouteTokens - 1) / kRouteTokens, chunk = t0 / kRouteTokens;
    const int n = min(per_block, T - t0), pairs = n * K;
    pdl_wait();
    pdl_trigger();
    uint4 v[kRowVecs];
    auto load = [&](int j) {
#pragma unroll
        for (int u = 0; u < kRowVecs; ++u) {
            const int i = 8 * (tid + kPlaceThreads * u);
            if (i < H) v[u] = ld_cg16(h + static_cast<int64_t>(t0 + j) * H + i);
        }
    };
    load(0);
    const int lanes = E <= 64 ? 64 : 128, e = tid & (lanes - 1);
    int all = 0, below = 0;
    if (e < E) {
#pragma unroll 8
        for (int c = tid / lanes; c < chunks; c += kPlaceThreads / lanes) {
            const int k = __ldcg(counts + c * E + e);
            all += k;
            below += c < chunk ? k : 0;
        }
    }
    s_all[tid] = all;
    s_below[tid] = below;
    __syncthreads();
    if (tid < 32) {  // four neighbouring experts a lane, then over the lanes
        int sum[4], mine = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = 4 * tid + i;
            sum[i] = 0;
            if (x < E)
                for (int u = x; u < kPlaceThreads; u += lanes) sum[i] += s_all[u];
            mine += sum[i];
        }
        int first = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, first, o);
            if (tid >= o) first += up;
        }
        first -= mine;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = 4 * tid + i;
            if (x < E) {
                int before = first;
                for (int u = x; u < kPlaceThreads; u += lanes) before += s_below[u];
                s_base[x] = before;
                if (blockIdx.x == 0) seg[x] = first;
            }
            first += sum[i];
        }
        if (blockIdx.x == 0 && tid == 31) seg[E] = first;
    }
    __syncthreads();
    for (int i = tid; i < pairs; i += kPlaceThreads) {
        const int64_t p = static_cast<int64_t>(t0) * K + i;
        const int row = s_base[__ldcg(top_i + p)] + __ldcg(rank + p);
        s_row[i] = row;
        place[p] = row;
    }
    __syncthreads();
    for (int j = 0; j < n; ++j) {
        uint4 w[kRowVecs];
#pragma unroll
        for (int u = 0; u < kRowVecs; ++u) w[u] = v[u];
        if (j + 1 < n) load(j + 1);
        for (int k = 0; k < K; ++k) {
            __half* dst = x_sorted + static_cast<int64_t>(s_row[j * K + k]) * H;
#pragma unroll
            for (int u = 0; u < kRowVecs; ++u) {
                const int i = 8 * (tid + kPlaceThreads * u);
                if (i < H) *reinterpret_cast<uint4*>(dst + i) = w[u];
            }
        }
    }
}

// out[t] = fp16(sum_k w[t, k] * y[place[t, k]]), products and sums in slot order in fp32, y not rounded before.
__global__ void __launch_bounds__(kRowThreads) weighted_sum_kernel(const float* __restrict__ y, const int32_t* __restrict__ place, const __half* __restrict__ top_w, int K,
                                                                   int H, __half* __restrict__ out) {
    pdl_wait();
    pdl_trigger();
    const int64_t t = blockIdx.x;
    for (int i = 4 * (threadIdx.x + kRowThreads * blockIdx.y); i < H; i += 4 * kRowThreads * gridDim.y) {
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < K; ++k) {
            const float w = __half2float(__ldg(top_w + t * K + k));
            const float4 v = __ldcg(reinterpret_cast<const float4*>(y + static_cast<int64_t>(__ldg(place + t * K + k)) * H + i));
            a[0] = fmaf(w, v.x, a[0]);
            a[1] = fmaf(w, v.y, a[1]);
            a[2] = fmaf(w, v.z, a[2]);
            a[3] = fmaf(w, v.w, a[3]);
        }
        __align__(8) __half o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = __float2half_rn(a[j]);
        *reinterpret_cast<uint2*>(out + t * H + i) = *reinterpret_cast<const uint2*>(o);
    }
}

__global__ void __launch_bounds__(kRowThreads) gather_rows_kernel(const __half* __restrict__ h, const int32_t* __restrict__ pair_of, int K, int H,
                                                                  __half* __restrict__ x_sorted) {
    pdl_wait();
    pdl_trigger();
    const int64_t r = blockIdx.x, t = pair_of[r] / K;
    for (int i = 8 * threadIdx.x; i < H; i += 8 * kRowThreads)
        *reinterpret_cast<uint4*>(x_sorted + r * H + i) = ld_cg16(h + t * H + i);
}

}  // namespace

int launch_embed_norm(const int64_t* tokens, const __half* embed, int64_t vocab, int T, int H, const __half* w, float eps, __half* x, __half* h, int* err,
                      const LaunchCfg& lc) {
    return launch_kernel(embed_norm_kernel, dim3(T), dim3(kRowThreads), 0, lc, tokens, embed, vocab, H, w, eps, x, h, err);
}

int launch_combine_norm(const __half* y, const int32_t* place, const float* top_w, int T, int K, const __half* x1, int H, const __half* w, float eps, __half* x2,
                        __half* h, const LaunchCfg& lc) {
    return launch_kernel(H <= 8 * kRowThreads ? combine_norm_kernel<1> : combine_norm_kernel<2>, dim3(T), dim3(kRowThreads), 0, lc, y, place, top_w, K, x1, H, w, eps, x2, h);
}

int launch_qkv_rows(const QkvRows& p, const LaunchCfg& lc) {
    const bool one = p.heads * 128 <= 8 * kRowThreads;
    auto* kernel = p.kc ? (one ? qkv_rows_kernel<true, 1> : qkv_rows_kernel<true, 2>) : (one ? qkv_rows_kernel<false, 1> : qkv_rows_kernel<false, 2>);
    return launch_kernel(kernel, dim3(p.T), dim3(kRowThreads), 0, lc, p);
}

int launch_norm_route(const __half* x, const __half* norm_w, float eps, const __half* router, int T, int H, int E, int top_k, int norm, __half* h, float* top_w,
                      int32_t* top_i, int32_t* rank, int32_t* counts, const LaunchCfg& lc) {
    const dim3 grid((T + kRouteTokens - 1) / kRouteTokens), block(kRouteWarps * 32);
    const size_t smem = std::max(static_cast<size_t>(kRouteWarps) * kRouteTokens * E * sizeof(float), static_cast<size_t>(kRouteTokens) * (H + 8) * sizeof(__half));
    auto run = [&](auto* kernel) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess) return set_error(LEMOQ_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(err));
        return launch_kernel(kernel, grid, block, smem, lc, x, norm_w, eps, router, T, H, E, top_k, norm, h, top_w, top_i, rank, counts);
    };
    if (H <= 2048) return E <= 64 ? run(norm_route_kernel<8, 8>) : run(norm_route_kernel<16, 8>);
    return E <= 64 ? run(norm_route_kernel<8, 16>) : run(norm_route_kernel<16, 16>);
}

// Tokens of a block: up to eight blocks an SM, and no more than that, because each of them reads all counts.  With more tokens than kPlaceTokens
// those reads (a block 256 bytes for 16 tokens, and one block for 16) outgrow the copies.
int launch_place_rows(const int32_t* top_i, const int32_t* rank, const int32_t* counts, int T, int K, int E, const __half* h, int H, int32_t* place, int32_t* seg,
                      __half* x_sorted, const LaunchCfg& lc) {
    int per = 1;
    while (per < kRouteTokens && T / per > 8 * sm_count()) per *= 2;
    return launch_kernel(place_rows_kernel, dim3((T + per - 1) / per), dim3(kPlaceThreads), 0, lc, top_i, rank, counts, T, K, E, h, H, per, place, seg, x_sorted);
}

template <typename ID>
static int plan_and_gather(const ID* ids, int P, int E, const __half* h, int K, int H, int32_t* place, int32_t* pair_of, int32_t* seg, __half* x_sorted, int* err,
                           const LaunchCfg& lc) {
    if (std::is_same<ID, int64_t>::value && P <= kGatherPairs)
        return launch_kernel(pair_plan_kernel<int64_t, true>, dim3(E), dim3(kPlanThreads), 0, lc, reinterpret_cast<const int64_t*>(ids), P, E, place, pair_of, seg, h, K, H, x_sorted, err);
    if (int rc = launch_kernel(pair_plan_kernel<ID, false>, dim3(E), dim3(kPlanThreads), 0, lc, ids, P, E, place, pair_of, seg, h, K, H, x_sorted, err)) return rc;
    return launch_kernel(gather_rows_kernel, dim3(P), dim3(kRowThreads), 0, lc, h, pair_of, K, H, x_sorted);
}

int launch_pairs(const int32_t* ids, int P, int E, const __half* h, int K, int H, int32_t* place, int32_t* pair_of, int32_t* seg, __half* x_sorted, int* err,
                 const LaunchCfg& lc) {
    return plan_and_gather(ids, P, E, h, K, H, place, pair_of, seg, x_sorted, err, lc);
}

int launch_pairs(const int64_t* ids, int P, int E, const __half* h, int K, int H, int32_t* place, int32_t* pair_of, int32_t* seg, __half* x_sorted, int* err,
                 const LaunchCfg& lc) {
    return plan_and_gather(ids, P, E, h, K, H, place, pair_of, seg, x_sorted, err, lc);
}

int launch_weighted_sum(const float* y, const int32_t* place, const __half* top_w, int T, int K, int H, __half* out, const LaunchCfg& lc) {
    return launch_kernel(weighted_sum_kernel, dim3(T, (H / 4 + kRowThreads - 1) / kRowThreads), dim3(kRowThreads), 0, lc, y, place, top_w, K, H, out);
}

}  // namespace lemoq
