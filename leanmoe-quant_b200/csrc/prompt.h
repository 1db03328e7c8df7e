// Launch interface of the kernels for many tokens at once (prompt_ops.cu, prompt_attn.cu).
#pragma once

#include "kernels.h"

namespace lemoq {

int launch_embed_norm(const int64_t* tokens, const __half* embed, int64_t vocab, int T, int H, const __half* w, float eps, __half* x, __half* h, int* err,
                      const LaunchCfg& lc);
int launch_combine_norm(const __half* y, const int32_t* place, const float* top_w, int T, int K, const __half* x1, int H, const __half* w, float eps, __half* x2,
                        __half* h, const LaunchCfg& lc);

struct QkvRows {
    const __half* qkv = nullptr;     // (T, 3A)
    const __half *q_norm = nullptr, *k_norm = nullptr;        // (A)
    const __half *rope_cos = nullptr, *rope_sin = nullptr;    // (S, 128)
    const int64_t* pos = nullptr;    // (T) cache slot of each row; with kc: one slot for all
    __half* q = nullptr;             // (T, A)
    __half *keys = nullptr, *values = nullptr;                // (heads, S, 128)
    int8_t *kc = nullptr, *vc = nullptr;                      // instead of keys / values: (T * heads, S, 128) codes ...
    __half *ks = nullptr, *vs = nullptr;                      // ... and (T * heads, S) scales
    float eps = 0.f;
    int T = 0, heads = 0, S = 0;
    int* err_flag = nullptr;
};
int launch_qkv_rows(const QkvRows& p, const LaunchCfg& lc);

// h = RMSNorm(x); logits fp16(h . router^T), softmax + top-k of every row.  E a multiple of 8, <= 128; H a multiple of 64, <= 4096.  Of the pairs of
// every 16 tokens also: counts (ceil(T / 16), E) by expert, and rank (T, top_k), the place of a pair among those of its expert.
int launch_norm_route(const __half* x, const __half* norm_w, float eps, const __half* router, int T, int H, int E, int top_k, int norm, __half* h, float* top_w,
                      int32_t* top_i, int32_t* rank, int32_t* counts, const LaunchCfg& lc);
// Stable sort of the pairs by expert from those: place[p] = row of pair p in expert order, seg[e] = first row of e, x_sorted[place[p]] = h[p / K].
constexpr int kPlaceTokens = 16384;  // at most
int launch_place_rows(const int32_t* top_i, const int32_t* rank, const int32_t* counts, int T, int K, int E, const __half* h, int H, int32_t* place, int32_t* seg,
                      __half* x_sorted, const LaunchCfg& lc);
// Stable sort of the P = T * K pairs by expert: place[p] = row of pair p in expert order, pair_of[row] = p, seg[e] = first row of e,
// x_sorted[row] = h[pair_of[row] / K].  Ids outside [0, E) are clamped and flagged.
int launch_pairs(const int32_t* ids, int P, int E, const __half* h, int K, int H, int32_t* place, int32_t* pair_of, int32_t* seg, __half* x_sorted, int* err,
                 const LaunchCfg& lc);
int launch_pairs(const int64_t* ids, int P, int E, const __half* h, int K, int H, int32_t* place, int32_t* pair_of, int32_t* seg, __half* x_sorted, int* err,
                 const LaunchCfg& lc);
int launch_weighted_sum(const float* y, const int32_t* place, const __half* top_w, int T, int K, int H, __half* out, const LaunchCfg& lc);

struct PromptAttn {
    const __half* q = nullptr;       // (T, heads * 128)
    const __half *keys = nullptr, *values = nullptr;  // (heads, S, 128)
    const int64_t* pos = nullptr;    // (T): row t sees slots [0, pos[t]]
    __half* out = nullptr;           // (T, heads * 128)
    int T = 0, heads = 0, S = 0;
    float scale = 0.f;
    int* err_flag = nullptr;
};
int launch_prompt_attn(const PromptAttn& p, const LaunchCfg& lc);

}  // namespace lemoq
