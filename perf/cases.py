"""What is timed when this framework is timed: the calls a user of it makes, over the range in which they are made.

Three jobs on the OLMoE-1B-7B architecture in the canonical form (W8A16 group 128 on attention, experts and lm_head), and
the operators of the kernel API that a model of one's own is patched together from:

decode     tokens of ONE sequence through a captured ``StaticCacheDecodeSession``: int8 or fp16 KV, any filled length, either
           chained on the device (``replay_chained``) or driven by the host token by token (``replay``)
prefill    the prompt of such a session (``StaticCacheDecodeSession.prefill``): what stands between a request and its first token
lockstep   one step of many sequences (``ExpertParallelDecoder`` on one GPU, captured)
linear     a W8 linear on one or some tokens (``QuantLinear``)
experts    the routed W8 experts on one or some tokens (``grouped_moe_forward_quant`` / ``_tokens``)
attention  one query row against an int8 or fp16 KV cache (``attn_decode_forward_int8`` / ``attn_decode_forward``)

Weights are random (nothing can be downloaded), but scaled so that the model behaves like a trained one where it matters
for a comparison: the residual stream is dominated by the embedding, the router is decisive, and the most likely next
token is clear (the lm_head rows are embedding rows in another order).  With plain N(0, 0.02) everywhere, the choice
between nearly equal experts and tokens hangs on the last bit of fp16 sums and two right implementations part ways.
"""

from __future__ import annotations

import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "leanmoe-quant_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from benchmarks.bytes import CANONICAL_QUANT, ModelSpec, byte_budget, weight_budget  # noqa: E402
from benchmarks.cudagraph import StaticCacheDecodeSession  # noqa: E402
from benchmarks.expert_parallel import ExpertParallelDecoder  # noqa: E402
from benchmarks.runner import install_replacements  # noqa: E402
from lemoq.kernels.attn_decode import attn_decode_forward, attn_decode_forward_int8  # noqa: E402
from lemoq.kernels.kv_int8 import kv_int8_bulk_quantize  # noqa: E402
from lemoq.kernels.moe_grouped_quant import grouped_moe_forward_quant, grouped_moe_forward_quant_tokens, quantize_fused_experts  # noqa: E402
from lemoq.kernels.moe_static import FusedExperts  # noqa: E402
from lemoq.model import OlmoeConfig, OlmoeForCausalLM  # noqa: E402
from lemoq.quant.linear import QuantLinear, SchemeSpec  # noqa: E402

DEV = "cuda"
GROUP = 128
SPEC = ModelSpec()  # 16 layers, hidden 2048, 16 heads x 128, 64 experts top-8 of width 1024, vocabulary 50304
H, A, F, E, K, V = SPEC.hidden, SPEC.num_attention_heads * SPEC.head_dim, SPEC.expert_ffn_dim, SPEC.num_experts, SPEC.top_k, SPEC.vocab
HEADS, DIM = SPEC.num_attention_heads, SPEC.head_dim
QUANT = {"bit_width": "w8a16", "dequant": "fused", "group_size": GROUP}


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a chat just begun: the smallest decode call, one token with a short cache, driven by the host (it reads the token)
        {"name": "decode-first-token", "kind": "decode", "layers": 16, "ctx": 48, "kv": "int8", "loop": "host", "steps": 1},
        # the headline of the benchmark: greedy tokens at 1024 cached positions, 32 per read-back
        {"name": "decode-1024", "kind": "decode", "layers": 16, "ctx": 1024, "kv": "int8", "loop": "device", "steps": 32},
        # the model's longest context
        {"name": "decode-4096", "kind": "decode", "layers": 16, "ctx": 4096, "kv": "int8", "loop": "device", "steps": 16},
        # the arm without KV quantisation, host-driven (a sampler on the host), at a length that no tile divides
        {"name": "decode-fp16-kv", "kind": "decode", "layers": 16, "ctx": 1537, "kv": "fp16", "loop": "host", "steps": 4},
        # time to first token: a one-line question, the benchmark's prompt length, and a full context
        {"name": "prefill-61", "kind": "prefill", "layers": 16, "ctx": 61},
        {"name": "prefill-1024", "kind": "prefill", "layers": 16, "ctx": 1024},
        {"name": "prefill-4096", "kind": "prefill", "layers": 16, "ctx": 4096},
        # offline batch: the lockstep configuration of the benchmark, and a small ragged batch
        {"name": "lockstep-64x2048", "kind": "lockstep", "layers": 16, "sequences": 64, "ctx": 2048},
        {"name": "lockstep-11x700", "kind": "lockstep", "layers": 16, "sequences": 11, "ctx": 700},
        # operators: the smallest linear of the model on one token, the expert layer on a small batch, attention over a long cache
        {"name": "linear-o_proj", "kind": "linear", "rows": 2048, "cols": 2048, "tokens": 1},
        {"name": "experts-16", "kind": "experts", "tokens": 16},
        {"name": "attention-4097", "kind": "attention", "filled": 4097, "kv": "int8"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """Drawn models are 2 to 6 layers deep (the runner's ``--layers``): depth only repeats the work of a layer, and a
    shallow model is built in a moment."""
    kind = rng.choice(["decode", "prefill", "lockstep", "linear", "experts", "attention"])
    if kind == "decode":
        return {"kind": kind, "layers": rng.choice([2, 3, 4, 6]), "ctx": _log_int(rng, 16, 4096), "kv": rng.choice(["int8", "int8", "fp16"]),
                "loop": rng.choice(["device", "host"]), "steps": _log_int(rng, 1, 32)}
    if kind == "prefill":
        return {"kind": kind, "layers": rng.choice([2, 3, 4, 6]), "ctx": _log_int(rng, 16, 4096)}
    if kind == "lockstep":
        return {"kind": kind, "layers": rng.choice([2, 3, 4, 6]), "sequences": _log_int(rng, 2, 64), "ctx": _log_int(rng, 64, 2048)}
    if kind == "linear":  # o_proj, packed q.k.v and lm_head shapes
        return {"kind": kind, "rows": rng.choice([2048, 6144, 50304]), "cols": 2048, "tokens": _log_int(rng, 1, 256)}
    if kind == "experts":
        return {"kind": kind, "tokens": _log_int(rng, 1, 64)}
    return {"kind": kind, "filled": _log_int(rng, 16, 4128), "kv": rng.choice(["int8", "fp16"])}


# ------------------------------------------------------------------------------------------------ what a program has in hand
def _generator(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + salt)


def _model(seed, layers, ctx, new_tokens):
    cfg = OlmoeConfig(num_hidden_layers=layers)
    with torch.device("meta"):  # the default initialisation would be thrown away
        model = OlmoeForCausalLM(cfg).to(torch.float16)
    model = model.to_empty(device=DEV).eval()
    g = _generator(seed)
    with torch.no_grad():
        for p in model.parameters():
            p.fill_(1.0) if p.dim() == 1 else p.normal_(0.0, cfg.initializer_range, generator=g)
        embed = model.model.embed_tokens.weight
        embed.mul_(1.0 / cfg.initializer_range)
        for layer in model.model.layers:
            layer.mlp.gate.weight.mul_(5.0)
        model.lm_head.weight.copy_(embed[torch.randperm(V, generator=g, device=DEV)] * cfg.initializer_range)
    install_replacements(model, attn="kernel", moe="grouped", quant_cfg=QUANT, rmsnorm="fused", ctx=ctx, max_new_tokens=new_tokens,
                         device=DEV)
    return model


def _prompt(seed, ctx):
    return torch.randint(0, V, (1, ctx), generator=_generator(seed, 1), device=DEV)


def _prepare_decode(case, seed):
    ctx, steps = case["ctx"], case["steps"]
    before = os.environ.get("LEMOQ_KV_INT8")
    os.environ["LEMOQ_KV_INT8"] = "1" if case["kv"] == "int8" else "0"  # the runner's switch, read when the step is captured
    try:
        session = StaticCacheDecodeSession(_model(seed, case["layers"], ctx, 32), _prompt(seed, ctx), ctx=ctx, max_new_tokens=32,
                                           device=DEV, engine="step")
        session.capture(warmup=1)
    finally:
        if before is None:
            del os.environ["LEMOQ_KV_INT8"]
        else:
            os.environ["LEMOQ_KV_INT8"] = before
    return {"session": session, "ctx": ctx, "steps": steps, "chained": case["loop"] == "device", "first": session.seed_token_id}


def _prepare_prefill(case, seed):
    session = StaticCacheDecodeSession(_model(seed, case["layers"], case["ctx"], 32), _prompt(seed, case["ctx"]), ctx=case["ctx"],
                                       max_new_tokens=32, device=DEV)
    return {"session": session}


def _prepare_lockstep(case, seed):
    model, n, ctx = _model(seed, case["layers"], case["ctx"], 32), case["sequences"], case["ctx"]
    session = StaticCacheDecodeSession(model, _prompt(seed, ctx), ctx=ctx, max_new_tokens=32, device=DEV, engine="ops")
    decoder = ExpertParallelDecoder(model, session, sequences=n, world=1, rank=0, static_exchange=True)
    decoder.capture()
    return {"decoder": decoder, "ctx": ctx, "tokens": torch.randint(0, V, (n,), generator=_generator(seed, 2), device=DEV)}


def _prepare_linear(case, seed):
    n, k, g = case["rows"], case["cols"], _generator(seed)
    dense = torch.nn.Linear(k, n, bias=False, device=DEV, dtype=torch.float16)
    with torch.no_grad():
        dense.weight.normal_(0.0, 0.02, generator=g)
    spec = SchemeSpec.from_flags("w8a16", GROUP, dequant="fused")
    return {"linear": QuantLinear(dense, spec), "x": torch.randn(1, case["tokens"], k, generator=g, device=DEV).half()}


def _prepare_experts(case, seed):
    g = _generator(seed)
    fused = FusedExperts(torch.empty(E, 2 * F, H, device=DEV, dtype=torch.float16).normal_(0.0, 0.02, generator=g),
                         torch.empty(E, H, F, device=DEV, dtype=torch.float16).normal_(0.0, 0.02, generator=g))
    x = torch.randn(case["tokens"], H, generator=g, device=DEV).half()
    weights, ids = torch.topk(torch.softmax(torch.randn(case["tokens"], E, generator=g, device=DEV), dim=-1), K, dim=-1)
    return {"experts": quantize_fused_experts(fused, group_size=GROUP), "x": x, "ids": ids, "weights": weights.half()}


def _prepare_attention(case, seed):
    g, room = _generator(seed), -(-case["filled"] // 32) * 32 + 32
    keys, values = (torch.randn(1, HEADS, room, DIM, generator=g, device=DEV).half() for _ in range(2))
    state = {"q": torch.randn(1, HEADS, 1, DIM, generator=g, device=DEV).half(), "kv": case["kv"],
             "filled": torch.tensor([case["filled"]], dtype=torch.int32, device=DEV)}
    state["cache"] = kv_int8_bulk_quantize(keys, values) if case["kv"] == "int8" else {"k": keys, "v": values}
    return state


_PREPARE = {"decode": _prepare_decode, "prefill": _prepare_prefill, "lockstep": _prepare_lockstep, "linear": _prepare_linear,
            "experts": _prepare_experts, "attention": _prepare_attention}


def prepare(case, seed):
    with torch.no_grad():
        state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _cache_of(session):
    return {"keys": [layer.keys for layer in session.cache.layers], "values": [layer.values for layer in session.cache.layers]}


def run(state):
    kind = state["kind"]
    if kind == "decode":  # from the prompt's end again: a second answer to the same prompt
        session = state["session"]
        session.set_position(state["ctx"])
        session.current_token_id = state["first"]
        if state["chained"]:
            tokens = session.replay_chained(state["steps"])
        else:
            tokens = []
            for _ in range(state["steps"]):
                session.replay()
                tokens.append(session.current_token_id)
        return {"tokens": torch.tensor(tokens), "logits": session.logits, **_cache_of(session)}
    if kind == "prefill":
        session = state["session"]
        output = session.prefill()
        return {"logits": output.logits, "token": session.current_token_id, **_cache_of(session)}
    if kind == "lockstep":
        decoder = state["decoder"]
        decoder.position = state["ctx"]
        return decoder.step(state["tokens"])
    with torch.no_grad():
        if kind == "linear":
            return state["linear"](state["x"])
        if kind == "experts":
            if state["x"].shape[0] == 1:
                return grouped_moe_forward_quant(state["x"][0], state["experts"], state["ids"][0], state["weights"][0])
            return grouped_moe_forward_quant_tokens(state["x"], state["experts"], state["ids"], state["weights"])
        cache = state["cache"]
        if state["kv"] == "int8":
            return attn_decode_forward_int8(state["q"], cache["kc"], cache["ks"], cache["vc"], cache["vs"], state["filled"])
        return attn_decode_forward(state["q"], cache["k"], cache["v"], state["filled"])


# ------------------------------------------------------------------------------------------------ what it cannot do without
def _w8(rows, cols):
    return rows * cols + rows * (cols // GROUP) * 2


def _distinct_experts(tokens):
    """Experts that ``tokens`` tokens reach between them when each picks 8 of 64 at random."""
    return E * (1.0 - (1.0 - K / E) ** tokens)


def _model_work(layers, tokens, kv_read, kv_written, attended):
    """``tokens`` rows through the model in one go: every weight that is needed read once, the embedding rows in, the
    logits of every row out, ``kv_read`` / ``kv_written`` bytes of cache, ``attended`` (row, position) pairs."""
    experts = _distinct_experts(tokens) * (_w8(2 * F, H) + _w8(H, F))
    layer = _w8(3 * A, H) + _w8(H, A) + E * H * 2 + experts
    flops = 2.0 * tokens * (layers * (4 * A * H + E * H + K * 3 * F * H) + H * V) + layers * 4.0 * A * attended
    return {"bytes": layers * layer + _w8(V, H) + tokens * (H + V) * 2 + kv_read + kv_written, "flops": flops}


def work(case):
    kind, layers = case["kind"], case.get("layers", 0)
    if kind == "decode":
        spec, total = ModelSpec(layers=layers), 0
        for step in range(case["steps"]):
            total += byte_budget(spec, case["ctx"] + step + 1, CANONICAL_QUANT, kv_int8=case["kv"] == "int8")["T"] + V * 2
        weights = weight_budget(spec, CANONICAL_QUANT)["total_bytes"] * case["steps"]
        return {"bytes": total, "flops": 2.0 * weights + 4.0 * layers * A * case["steps"] * (case["ctx"] + case["steps"] / 2)}
    if kind == "prefill":
        ctx = case["ctx"]
        return _model_work(layers, ctx, 0, layers * 2 * ctx * A * 2, ctx * (ctx + 1) / 2)
    if kind == "lockstep":
        n, ctx = case["sequences"], case["ctx"]
        row = layers * 2 * HEADS * (DIM + 2)
        return _model_work(layers, n, n * ctx * row, n * row, n * (ctx + 1))
    if kind == "linear":
        n, k, t = case["rows"], case["cols"], case["tokens"]
        return {"bytes": _w8(n, k) + t * (n + k) * 2, "flops": 2.0 * n * k * t}
    if kind == "experts":
        t = case["tokens"]
        return {"bytes": _distinct_experts(t) * (_w8(2 * F, H) + _w8(H, F)) + 2 * t * H * 2, "flops": 2.0 * t * K * 3 * F * H}
    per_position = 2 * HEADS * (DIM + 2 if case["kv"] == "int8" else 2 * DIM)
    return {"bytes": case["filled"] * per_position + 2 * HEADS * DIM * 2, "flops": 4.0 * A * case["filled"]}


def tolerance(case):
    """fp16 activations and outputs, fp32 sums: 2e-3 for one operator; through the layers of the model the roundings of
    fp16 activations add up, and now and then the eighth expert of a token is another, nearly equal one."""
    if case["kind"] in ("decode", "prefill", "lockstep"):
        return {"rel": 1e-2}
    return {"rel": 2e-3}
