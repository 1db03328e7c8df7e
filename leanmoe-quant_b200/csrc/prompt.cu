// Many tokens through the whole model, all layers, logits of every row:
//   lemoq_prompt_run    a prompt: T rows of one sequence, K/V rows left in its fp16 caches, causal attention over them
//   lemoq_lockstep_run  one token of each of T sequences, all at the same slot: K/V rows quantised into each sequence's int8 caches,
//                       decode attention over those
//
// Nine kernels per layer, launched from here with programmatic dependent launch: the prompt of a short question is
// bound by the 6.9 GB of weights all experts together have (1.1 ms), so a launch gap or a host call per expert is what it
// must not pay; a long prompt is bound by the tensor cores (w8_gemm.cu, prompt_attn.cu); a lockstep step by the weights and its
// sequences' caches (attn_i8.cu).
#include <algorithm>

#include "prompt.h"

namespace lemoq {
namespace {

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

struct PromptBuffers {
    __half *x, *x1, *h, *qkv, *q, *ctx, *pairs, *act;
    float* top_w;
    int32_t *top_i, *place, *pair_of, *seg, *counts;
};

size_t carve_prompt(const lemoq_step_desc& d, int T, char* base, PromptBuffers* b) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* at = base + off;
        off += up256(bytes);
        return at;
    };
    const size_t t = T, A = static_cast<size_t>(d.heads) * d.head_dim, P = t * d.top_k;
    PromptBuffers o;
    o.x = reinterpret_cast<__half*>(take(2 * t * d.hidden));
    o.x1 = reinterpret_cast<__half*>(take(2 * t * d.hidden));
    o.h = reinterpret_cast<__half*>(take(2 * t * d.hidden));
    o.qkv = reinterpret_cast<__half*>(take(2 * t * 3 * A));
    o.q = reinterpret_cast<__half*>(take(2 * t * A));
    o.ctx = reinterpret_cast<__half*>(take(2 * t * A));
    o.pairs = reinterpret_cast<__half*>(take(2 * P * d.hidden));  // the experts' inputs, then their outputs
    o.act = reinterpret_cast<__half*>(take(2 * P * d.ffn));
    o.top_w = reinterpret_cast<float*>(take(4 * P));
    o.top_i = reinterpret_cast<int32_t*>(take(4 * P));
    o.place = reinterpret_cast<int32_t*>(take(4 * P));
    o.pair_of = reinterpret_cast<int32_t*>(take(4 * P));  // norm_route's ranks, then (very many tokens) the pair of a row
    o.seg = reinterpret_cast<int32_t*>(take(4 * (static_cast<size_t>(d.experts) + 1)));
    o.counts = reinterpret_cast<int32_t*>(take(4 * ((t + 15) / 16) * d.experts));
    if (b) *b = o;
    return off;
}

int validate_prompt(const lemoq_step_desc& d) {
    LEMOQ_REQUIRE(d.layers > 0 && d.hidden > 0 && d.heads > 0 && d.experts > 0 && d.top_k > 0 && d.ffn > 0 && d.vocab > 0 && d.max_len > 0,
                  LEMOQ_ERR_INVALID, "prompt: all sizes must be positive");
    LEMOQ_REQUIRE(d.head_dim == 128, LEMOQ_ERR_UNSUPPORTED, "prompt: head_dim must be 128");
    LEMOQ_REQUIRE(d.hidden % 128 == 0 && d.hidden <= 4096 && d.heads <= 32 && d.ffn % 128 == 0, LEMOQ_ERR_UNSUPPORTED,
                  "prompt: hidden and ffn must be multiples of 128, hidden and heads * 128 at most 4096");
    LEMOQ_REQUIRE(d.experts % 8 == 0 && d.experts <= 128 && d.top_k <= 32 && d.top_k <= d.experts, LEMOQ_ERR_UNSUPPORTED,
                  "prompt: experts must be a multiple of 8, at most 128, top_k at most 32");
    LEMOQ_REQUIRE(d.group_size > 0 && d.group_size % 128 == 0 && d.hidden % d.group_size == 0 && d.ffn % d.group_size == 0 &&
                      d.heads * 128 % d.group_size == 0,
                  LEMOQ_ERR_UNSUPPORTED, "prompt: group_size must be a multiple of 128 that divides every row");
    return LEMOQ_OK;
}

}  // namespace
}  // namespace lemoq

using namespace lemoq;

namespace {

constexpr int kLockstepSplits = 16;  // at most (two or three sequences: 32 heads and few SMs busy without splits)
size_t attn_scratch_bytes(int heads) { return lemoq_attn_workspace_bytes(heads, 128, kLockstepSplits); }

// `filled` == nullptr: a prompt, positions (T).  Otherwise a lockstep step, positions and filled are device scalars.
int run_rows(const lemoq_step_desc* desc, const lemoq_layer_desc* layers, const int64_t* tokens, const int64_t* positions, const int32_t* filled, int T, void* logits,
             void* workspace, size_t workspace_bytes, int* err_flag, void* stream) {
    LEMOQ_REQUIRE(desc && layers && tokens && logits && workspace, LEMOQ_ERR_INVALID, "prompt: null pointer");
    const lemoq_step_desc& d = *desc;
    if (int rc = validate_prompt(d)) return rc;
    LEMOQ_REQUIRE(T > 0 && static_cast<int64_t>(T) * d.top_k <= (1 << 24), LEMOQ_ERR_INVALID, "prompt: T=%d out of range", T);
    LEMOQ_REQUIRE(d.embed && d.final_norm && d.lm_head_codes && d.lm_head_scale && d.rope_cos && d.rope_sin, LEMOQ_ERR_INVALID,
                  "prompt: null pointer in descriptor");
    const bool lockstep = filled != nullptr;
    for (const void* p : {d.embed, d.final_norm, static_cast<const void*>(d.lm_head_codes), d.lm_head_scale, d.rope_cos, d.rope_sin})
        LEMOQ_REQUIRE(aligned16(p), LEMOQ_ERR_INVALID, "prompt: unaligned pointer in descriptor");
    for (int i = 0; i < d.layers; ++i) {
        const lemoq_layer_desc& L = layers[i];
        const bool caches = lockstep ? L.kc && L.ks && L.vc && L.vs && aligned16(L.kc) && aligned16(L.vc) : L.keys && L.values && aligned16(L.keys) && aligned16(L.values);
        LEMOQ_REQUIRE(weights_placed(L) && caches, LEMOQ_ERR_INVALID, "prompt: null or unaligned pointer in layer %d", i);
    }
    LEMOQ_REQUIRE(aligned16(logits) && aligned16(workspace), LEMOQ_ERR_INVALID, "prompt: logits and workspace must be 16-byte aligned");
    PromptBuffers b;
    const size_t rows_bytes = carve_prompt(d, T, static_cast<char*>(workspace), &b), need = rows_bytes + (lockstep ? attn_scratch_bytes(T * d.heads) : 0);
    LEMOQ_REQUIRE(workspace_bytes >= need, LEMOQ_ERR_INVALID, "prompt: workspace of %zu bytes, needs %zu", workspace_bytes, need);
    if (!err_flag) err_flag = status_word();

    LaunchCfg lc;
    lc.stream = static_cast<cudaStream_t>(stream);
    LaunchCfg chained = lc;
    chained.pdl = true;
    auto half = [](const void* p) { return reinterpret_cast<const __half*>(p); };
    const int A = d.heads * 128, P = T * d.top_k;

    auto gemm = [&](const __half* x, int rows, const int8_t* codes, const void* scale, int N, int K, const __half* resid, __half* y) {
        W8GemmParams g;
        g.x = x; g.T = rows; g.codes = codes; g.scale = half(scale); g.N = N; g.K = K; g.group_size = d.group_size;
        g.resid = resid; g.y = y; g.exact = lockstep; g.err_flag = err_flag;
        return launch_w8_gemm(g, chained);
    };
#define LEMOQ_TRY(call)            \
    do {                           \
        if (int rc_ = (call)) return rc_; \
    } while (0)

    LEMOQ_TRY(launch_embed_norm(tokens, half(d.embed), d.vocab, T, d.hidden, half(layers[0].ln1), d.eps, b.x, b.h, err_flag, lc));
    for (int i = 0; i < d.layers; ++i) {
        const lemoq_layer_desc& L = layers[i];
        LEMOQ_TRY(gemm(b.h, T, L.qkv_codes, L.qkv_scale, 3 * A, d.hidden, nullptr, b.qkv));
        QkvRows r;
        r.qkv = b.qkv; r.q_norm = half(L.q_norm); r.k_norm = half(L.k_norm); r.rope_cos = half(d.rope_cos); r.rope_sin = half(d.rope_sin);
        r.pos = positions; r.q = b.q;
        if (lockstep) {
            r.kc = L.kc; r.vc = L.vc; r.ks = reinterpret_cast<__half*>(L.ks); r.vs = reinterpret_cast<__half*>(L.vs);
        } else {
            r.keys = reinterpret_cast<__half*>(L.keys); r.values = reinterpret_cast<__half*>(L.values);
        }
        r.eps = d.eps; r.T = T; r.heads = d.heads; r.S = d.max_len; r.err_flag = err_flag;
        LEMOQ_TRY(launch_qkv_rows(r, chained));
        if (lockstep) {
            AttnParams a;
            a.q = b.q; a.k = L.kc; a.v = L.vc; a.ks = r.ks; a.vs = r.vs; a.kv_head_stride = static_cast<int64_t>(d.max_len) * 128; a.filled = filled; a.out = b.ctx;
            a.heads = T * d.heads; a.S = d.max_len; a.D = 128; a.num_splits = std::min(kLockstepSplits, (2 * sm_count() + a.heads - 1) / a.heads);
            a.qk_scale_log2 = 1.4426950408889634f / sqrtf(128.0f); a.err_flag = err_flag;
            char* scratch = static_cast<char*>(workspace) + rows_bytes;
            a.counters = reinterpret_cast<unsigned int*>(scratch);
            a.part = reinterpret_cast<float*>(scratch + up256(sizeof(unsigned int) * a.heads));
            LEMOQ_REQUIRE(attn_i8_eligible(a), LEMOQ_ERR_UNSUPPORTED, "lockstep: %d sequences x %d heads x %d slots are too many", T, d.heads, d.max_len);
            LEMOQ_TRY(launch_attn_i8(a, chained));
        } else {
            PromptAttn a;
            a.q = b.q; a.keys = half(L.keys); a.values = half(L.values); a.pos = positions; a.out = b.ctx;
            a.T = T; a.heads = d.heads; a.S = d.max_len; a.scale = 1.0f / sqrtf(128.0f); a.err_flag = err_flag;
            LEMOQ_TRY(launch_prompt_attn(a, chained));
        }
        LEMOQ_TRY(gemm(b.ctx, T, L.o_codes, L.o_scale, d.hidden, A, b.x, b.x1));
        LEMOQ_TRY(launch_norm_route(b.x1, half(L.ln2), d.eps, half(L.router), T, d.hidden, d.experts, d.top_k, d.norm_topk_prob, b.h, b.top_w, b.top_i, b.pair_of, b.counts, chained));
        if (T <= kPlaceTokens)
            LEMOQ_TRY(launch_place_rows(b.top_i, b.pair_of, b.counts, T, d.top_k, d.experts, b.h, d.hidden, b.place, b.seg, b.pairs, chained));
        else
            LEMOQ_TRY(launch_pairs(b.top_i, P, d.experts, b.h, d.top_k, d.hidden, b.place, b.pair_of, b.seg, b.pairs, nullptr, chained));
        W8GemmParams g;
        g.x = b.pairs; g.T = P; g.codes = L.gu_codes; g.scale = half(L.gu_scale); g.N = 2 * d.ffn; g.K = d.hidden; g.group_size = d.group_size;
        g.seg = b.seg; g.E = d.experts; g.gate_up = true; g.y = b.act; g.exact = lockstep; g.err_flag = err_flag;
        LEMOQ_TRY(launch_w8_gemm(g, chained));
        g.x = b.act; g.codes = L.dn_codes; g.scale = half(L.dn_scale); g.N = d.hidden; g.K = d.ffn; g.gate_up = false; g.y = b.pairs;
        LEMOQ_TRY(launch_w8_gemm(g, chained));
        LEMOQ_TRY(launch_combine_norm(b.pairs, b.place, b.top_w, T, d.top_k, b.x1, d.hidden,
                                      half(i + 1 < d.layers ? layers[i + 1].ln1 : d.final_norm), d.eps, b.x, b.h, chained));
    }
    LEMOQ_TRY(gemm(b.h, T, d.lm_head_codes, d.lm_head_scale, d.vocab, d.hidden, nullptr, reinterpret_cast<__half*>(logits)));
    return LEMOQ_OK;
}

struct MoeBuffers {
    __half *x, *act;
    float* y;
    int32_t *place, *pair_of, *seg;
};

size_t carve_moe(int T, int K, int E, int H, int F, char* base, MoeBuffers* b) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* at = base + off;
        off += up256(bytes);
        return at;
    };
    const size_t P = static_cast<size_t>(T) * K;
    MoeBuffers o;
    o.x = reinterpret_cast<__half*>(take(2 * P * H));
    o.act = reinterpret_cast<__half*>(take(2 * P * F));
    o.y = reinterpret_cast<float*>(take(4 * P * H));
    o.place = reinterpret_cast<int32_t*>(take(4 * P));
    o.pair_of = reinterpret_cast<int32_t*>(take(4 * P));
    o.seg = reinterpret_cast<int32_t*>(take(4 * (static_cast<size_t>(E) + 1)));
    if (b) *b = o;
    return off;
}

}  // namespace

extern "C" size_t lemoq_moe_tokens_workspace_bytes(int T, int K, int E, int H, int F) {
    if (T <= 0 || K <= 0 || E <= 0 || H <= 0 || F <= 0) return 0;
    return carve_moe(T, K, E, H, F, nullptr, nullptr);
}

extern "C" int lemoq_moe_tokens_w8(const void* x, const int8_t* gu_codes, const void* gu_scale, const int8_t* dn_codes, const void* dn_scale, const int64_t* ids,
                                   const void* top_w, int T, int K, int E, int H, int F, int group_size, void* out, void* workspace, size_t workspace_bytes,
                                   int* err_flag, void* stream) {
    LEMOQ_REQUIRE(T >= 0 && K > 0 && E > 0 && H > 0 && F > 0, LEMOQ_ERR_INVALID, "moe_tokens_w8: bad shape");
    LEMOQ_REQUIRE(static_cast<int64_t>(T) * K <= (1 << 24) && E <= kMaxExperts, LEMOQ_ERR_UNSUPPORTED, "moe_tokens_w8: T=%d x K=%d pairs or E=%d experts above the limit", T, K, E);
    LEMOQ_REQUIRE(H % 128 == 0 && F % 128 == 0, LEMOQ_ERR_UNSUPPORTED, "moe_tokens_w8: hidden and ffn must be multiples of 128");
    LEMOQ_REQUIRE(group_size > 0 && group_size % 128 == 0 && H % group_size == 0 && F % group_size == 0, LEMOQ_ERR_UNSUPPORTED,
                  "moe_tokens_w8: group_size=%d must be a multiple of 128 that divides hidden and ffn", group_size);
    if (T == 0) return LEMOQ_OK;
    LEMOQ_REQUIRE(x && gu_codes && gu_scale && dn_codes && dn_scale && ids && top_w && out && workspace, LEMOQ_ERR_INVALID, "moe_tokens_w8: null pointer");
    LEMOQ_REQUIRE(aligned16(x) && aligned16(gu_codes) && aligned16(dn_codes) && aligned16(out) && aligned16(workspace), LEMOQ_ERR_INVALID,
                  "moe_tokens_w8: pointers must be 16-byte aligned");
    MoeBuffers b;
    const size_t need = carve_moe(T, K, E, H, F, static_cast<char*>(workspace), &b);
    LEMOQ_REQUIRE(workspace_bytes >= need, LEMOQ_ERR_INVALID, "moe_tokens_w8: workspace of %zu bytes, needs %zu", workspace_bytes, need);
    if (!err_flag) err_flag = status_word();
    LaunchCfg lc;
    lc.stream = static_cast<cudaStream_t>(stream);
    LaunchCfg chained = lc;
    chained.pdl = true;
    LEMOQ_TRY(launch_pairs(ids, T * K, E, reinterpret_cast<const __half*>(x), K, H, b.place, b.pair_of, b.seg, b.x, err_flag, lc));
    W8GemmParams g;
    g.x = b.x; g.T = T * K; g.codes = gu_codes; g.scale = reinterpret_cast<const __half*>(gu_scale); g.N = 2 * F; g.K = H; g.group_size = group_size;
    g.seg = b.seg; g.E = E; g.gate_up = true; g.y = b.act; g.err_flag = err_flag;
    LEMOQ_TRY(launch_w8_gemm(g, chained));
    g.x = b.act; g.codes = dn_codes; g.scale = reinterpret_cast<const __half*>(dn_scale); g.N = H; g.K = F; g.gate_up = false; g.y = nullptr; g.y32 = b.y;
    LEMOQ_TRY(launch_w8_gemm(g, chained));
    return launch_weighted_sum(b.y, b.place, reinterpret_cast<const __half*>(top_w), T, K, H, reinterpret_cast<__half*>(out), chained);
}
#undef LEMOQ_TRY

extern "C" size_t lemoq_prompt_workspace_bytes(const lemoq_step_desc* desc, int T) {
    if (!desc || T <= 0 || validate_prompt(*desc) != LEMOQ_OK) return 0;
    return carve_prompt(*desc, T, nullptr, nullptr);
}

extern "C" int lemoq_prompt_run(const lemoq_step_desc* desc, const lemoq_layer_desc* layers, const int64_t* tokens, const int64_t* positions, int T, void* logits,
                                void* workspace, size_t workspace_bytes, int* err_flag, void* stream) {
    LEMOQ_REQUIRE(positions, LEMOQ_ERR_INVALID, "prompt: null pointer");
    return run_rows(desc, layers, tokens, positions, nullptr, T, logits, workspace, workspace_bytes, err_flag, stream);
}

extern "C" size_t lemoq_lockstep_workspace_bytes(const lemoq_step_desc* desc, int T) {
    const size_t rows = lemoq_prompt_workspace_bytes(desc, T);
    return rows ? rows + attn_scratch_bytes(T * desc->heads) : 0;
}

extern "C" int lemoq_lockstep_run(const lemoq_step_desc* desc, const lemoq_layer_desc* layers, const int64_t* tokens, const int64_t* position,
                                  const int32_t* filled, int T, void* logits, void* workspace, size_t workspace_bytes, int* err_flag, void* stream) {
    LEMOQ_REQUIRE(position && filled, LEMOQ_ERR_INVALID, "lockstep: null pointer");
    return run_rows(desc, layers, tokens, position, filled, T, logits, workspace, workspace_bytes, err_flag, stream);
}
