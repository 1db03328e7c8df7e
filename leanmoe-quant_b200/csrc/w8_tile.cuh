// What the two forms of the W8 GEMM share (w8_gemm.cu: exact, w8_pair.cu: scaled): the call's shape, widening of codes, the group
// scales of a weight row, SwiGLU.
#pragma once

#include "tc.cuh"

namespace lemoq {

// What both kernels are told about a call.
struct W8Shape {
    int T, N, K, group, E, gate_up;
    const int32_t* seg;    // (E + 1) or null: one segment [0, T)
    const __half* scale;   // (E, N, K / group)
    const __half* resid;   // (T, N) or null
    __half* y;             // (T, N), or (T, N / 2) in gate/up mode
    float* y32;            // or, in the exact form: (T, N) in fp32
    int* err_flag;
    int scale_vecs;        // 16-byte vectors of a row's scales when they fit the shared rows (1 or 2), else 0
    int parts;             // exact form, SPLIT: blocks of a cluster that share a tile's groups
    int wide;              // scaled form: rows of y (and resid) begin on 16 bytes, eight values a store
    int cap;               // scaled form: most tokens of a tile, a multiple of 32
    int stages;            // and how many of its stages fit
};

struct Tile {
    int row0, row1;    // first weight row of the two M tiles inside the expert
    int e, t0, n;      // expert, first token, tokens
};

// One warp: tokens and tiles before each expert, for `mt` tiles along the weight rows and `cap` tokens (a power of two or a multiple of 32)
// along the tokens.
__device__ __forceinline__ void fill_tiles(const W8Shape& p, int cap, int mt, int* s_first, int* s_tok, int lane) {
    int carry = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
        const int e = e0 + lane;
        int a = 0, b = 0;
        if (e < p.E) {
            a = p.seg ? min(max(p.seg[e], 0), p.T) : 0;
            b = p.seg ? min(max(p.seg[e + 1], a), p.T) : p.T;
            s_tok[e] = a;
            if (e == p.E - 1) s_tok[p.E] = b;
        }
        const int mine = (b - a + cap - 1) / cap * mt;
        int v = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += up;
        }
        if (e < p.E) s_first[e] = carry + v - mine;
        carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) s_first[p.E] = carry;
}

// Tiles before expert e: first[e].  A tile number -> expert by binary search, then (tile along the rows, token tile): neighbours in
// the order share their weight rows and meet in L2.  The tokens of an expert are split evenly, in steps of `unit` (which divides cap, so no tile
// is empty).  row0 comes back as the tile's number along the rows.
__device__ __forceinline__ Tile find_tile(int i, const int* first, const int* tok, int E, int cap, int unit) {
    if (i >= first[E]) return Tile{0, 0, 0, 0, 0};
    int lo = 0, hi = E;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= i) lo = mid; else hi = mid;
    }
    Tile t;
    t.e = lo;
    const int cnt = tok[lo + 1] - tok[lo], nt = (cnt + cap - 1) / cap, r = i - first[lo], m = r / nt, b = r - m * nt;
    const int per = ((cnt + nt - 1) / nt + unit - 1) / unit * unit;
    t.t0 = tok[lo] + b * per;
    t.n = max(0, min(per, tok[lo + 1] - t.t0));
    t.row0 = t.row1 = m;
    return t;
}

// silu(gate) * up of two pairs, for fp16 results: exp and the quotients to about 2^-21, one reciprocal for both.  Below -43 the exponential is
// held at e^43 (its square is finite): such a gate gives less than 1e-12 whatever `up` is.  (With expf and rounded divisions the epilogue of a
// gate/up tile of 128 tokens took 9900 cycles, half as long as its MMAs.)
__device__ __forceinline__ void swiglu2(float g0, float u0, float g1, float u1, float& y0, float& y1) {
    const float a = 1.0f + __expf(-fmaxf(g0, -43.f)), b = 1.0f + __expf(-fmaxf(g1, -43.f)), r = __fdividef(1.0f, a * b);
    y0 = g0 * (r * b) * u0;
    y1 = g1 * (r * a) * u1;
}

// 16 codes -> 8 words of two exact fp16 each: bytes with the sign flipped dropped into 0x64__ are 1024 + 128 + c.
template <bool SCALED>
__device__ __forceinline__ void widen16(const uint4& w, __half scale, uint32_t* out) {
    const uint32_t u[4] = {w.x ^ 0x80808080u, w.y ^ 0x80808080u, w.z ^ 0x80808080u, w.w ^ 0x80808080u};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        __half2 a = codes_half2(u[i], 0x4140), b = codes_half2(u[i], 0x4342);
        if (SCALED) {
            a = __hmul2(a, __half2half2(scale));
            b = __hmul2(b, __half2half2(scale));
        }
        out[2 * i] = *reinterpret_cast<const uint32_t*>(&a);
        out[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&b);
    }
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Per device and idempotent; not a stream operation, so legal under capture.
template <typename K>
int allow_smem(K kernel, size_t bytes) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    return err == cudaSuccess ? LEMOQ_OK : set_error(LEMOQ_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(err));
}

int launch_w8_pair(W8Shape p, const __half* x, const int8_t* codes, const LaunchCfg& lc);

}  // namespace lemoq
