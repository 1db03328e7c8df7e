"""Many tokens through the whole model in one native call, for models in the canonical W8 form: a prompt (``lemoq_prompt_run``), or one
token of each of many sequences (``lemoq_lockstep_run``).

The module tree's own forward stays the path of everything else; :func:`run_prompt`, :func:`lockstep_plan` and :func:`run_lockstep` return
None for what the native path does not take.  The model is read anew at every call, as its modules' forwards would read it: nothing of a
call is kept for the next by the address or identity of a tensor or module.
"""

from __future__ import annotations

from array import array
from typing import Any, NamedTuple

import torch
import torch.nn.functional as F

from lemoq import _cabi

_PLAN = "_lemoq_prompt_plan"  # on the cache object: what the last native call over that cache was given

# the weights of a layer, in the order of ``LayerDesc``; behind them come the cache tensors
_LAYER_WEIGHTS = ("ln1", "ln2", "q_norm", "k_norm", "qkv_codes", "qkv_scale", "o_codes", "o_scale", "router", "gu_codes", "gu_scale", "dn_codes", "dn_scale")
_CACHES = ("keys", "values", "kc", "ks", "vc", "vs")
assert _LAYER_WEIGHTS + _CACHES == tuple(name for name, _ in _cabi.LayerDesc._fields_)


class Weights(NamedTuple):
    """The tensors of a model in the canonical form."""

    own: dict      # field of ``StepDesc`` -> tensor
    layers: list   # per layer, in the order of ``_LAYER_WEIGHTS``

    def tensors(self) -> list:
        return [*self.own.values(), *(t for layer in self.layers for t in layer)]


def read_weights(model: Any) -> Weights | None:
    """The tensors that the model's forwards would use now; None when a piece is not in the form the native path knows.  (Through the
    modules' own dictionaries: 300 attribute look-ups of ``nn.Module`` would take longer than the launches of a short prompt.)"""
    from lemoq.kernels.attn_decode import _decode_forward_impl
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts
    from lemoq.model import OlmoeAttention, OlmoeDecoderLayer
    from lemoq.quant.linear import QuantLinear

    m, lm = model.model, model.lm_head
    if type(lm) is not QuantLinear or lm.bias is not None or model.config.clip_qkv is not None or not len(m.layers):
        return None
    layers = []
    for layer in m.layers:
        if type(layer) is not OlmoeDecoderLayer:
            return None
        parts = layer._modules
        attn, mlp = parts["self_attn"], parts["mlp"]
        inner, here, moe = attn._modules, attn.__dict__, mlp.__dict__
        packed, o_proj, stacks = here.get("_lemoq_packed_qkv"), inner.get("o_proj"), moe.get("_static_experts")
        if (packed is None or type(o_proj) is not QuantLinear or o_proj._buffers["bias"] is not None or not isinstance(stacks, QuantFusedExperts)
                or getattr(here.get("forward"), "__func__", None) is not _decode_forward_impl
                or getattr(here.get("_lemoq_original_forward"), "__func__", None) is not OlmoeAttention.forward
                or here["num_key_value_groups"] != 1 or moe["_static_act"] not in (None, F.silu)):
            return None
        norms = [norm._parameters.get("weight") for norm in (parts["input_layernorm"], parts["post_attention_layernorm"], inner["q_norm"], inner["k_norm"])]
        if any(t is None for t in norms):
            return None
        layers.append((*norms, packed.packed, packed.scale, o_proj._buffers["packed"], o_proj._buffers["scale"], moe["_static_router"].contiguous(),
                       stacks.packed_gate_up, stacks.scale_gate_up, stacks.packed_down, stacks.scale_down))
    return Weights({"embed": m.embed_tokens.weight, "final_norm": m.norm.weight, "lm_head_codes": lm.packed, "lm_head_scale": lm.scale}, layers)


def describe(model: Any, weights: Weights, max_len: int, caches: list[dict]) -> tuple[Any, Any]:
    """``(StepDesc, LayerDesc array)`` of the model over one set of cache tensors per layer (named as in ``LayerDesc``): pointers only, the
    caller keeps the tensors for as long as the C side may read them."""
    cfg, m = model.config, model.model
    cos, sin = m.rotary_emb.tables(max_len, torch.float16, m.embed_tokens.weight.device)
    words = array("Q")
    for layer, slots in zip(weights.layers, caches):
        words.extend([t.data_ptr() for t in layer])
        words.extend([0 if slots.get(name) is None else slots[name].data_ptr() for name in _CACHES])
    desc = _cabi.StepDesc()
    desc.layers, desc.hidden, desc.heads, desc.head_dim = len(m.layers), cfg.hidden_size, cfg.num_attention_heads, cfg.head_dim
    desc.experts, desc.top_k, desc.ffn, desc.vocab = cfg.num_experts, cfg.num_experts_per_tok, cfg.intermediate_size, cfg.vocab_size
    desc.group_size, desc.max_len, desc.eps = int(model.lm_head.group_size), max_len, float(cfg.rms_norm_eps)
    desc.norm_topk_prob = int(bool(cfg.norm_topk_prob))
    for name, t in weights.own.items():
        setattr(desc, name, t.data_ptr())
    desc.rope_cos, desc.rope_sin = cos.data_ptr(), sin.data_ptr()
    return desc, (_cabi.LayerDesc * len(m.layers)).from_buffer(words)


def run_prompt(model: Any, input_ids: Any, cache: Any, cache_position: Any, position_ids: Any) -> Any:
    """Logits ``(1, T, V)`` of the prompt ``input_ids (1, T)``, with its K/V rows written into ``cache`` - or None when the
    model, the cache or the call is not of the kind the native path takes."""
    from lemoq.model import StaticCache

    weight = model.model.embed_tokens.weight
    if (torch.is_grad_enabled() or type(cache) is not StaticCache or input_ids.shape[0] != 1 or not weight.is_cuda or weight.dtype != torch.float16
            or input_ids.dtype != torch.int64 or cache_position.dtype != torch.int64 or not cache_position.is_cuda or cache_position.numel() != input_ids.shape[1]
            or position_ids.data_ptr() != cache_position.data_ptr() or position_ids.numel() != cache_position.numel() or not cache_position.is_contiguous()
            or len(cache.layers) != len(model.model.layers) or not _cabi.available()):
        return None
    weights = read_weights(model)
    if weights is None:
        return None
    cfg, device = model.config, weight.device
    for slot in cache.layers:
        if not slot.is_initialized:
            slot.lazy_initialization(torch.empty((1, cfg.num_attention_heads, 1, cfg.head_dim), dtype=torch.float16, device=device))
    desc, layers = describe(model, weights, cache.max_cache_len, [{"keys": s.keys, "values": s.values} for s in cache.layers])
    tokens = int(input_ids.shape[1])
    size = int(_cabi.lib().lemoq_prompt_workspace_bytes(desc, tokens))
    if size == 0:
        return None
    plan = cache.__dict__.setdefault(_PLAN, {})
    if plan.get("flags") is None:
        plan["flags"] = torch.zeros(1, dtype=torch.int32, device=device)
    ids = input_ids.contiguous()
    logits = torch.empty((1, tokens, cfg.vocab_size), dtype=torch.float16, device=device)
    workspace = torch.empty(size, dtype=torch.uint8, device=device)
    _cabi.call("lemoq_prompt_run", desc, layers, _cabi.ptr(ids), _cabi.ptr(cache_position), tokens, _cabi.ptr(logits),
               _cabi.ptr(workspace), size, _cabi.ptr(plan["flags"]), _cabi.current_stream(device))
    return logits


def lockstep_plan(model: Any, kv: list[dict], sequences: int, max_len: int) -> dict | None:
    """What :func:`run_lockstep` keeps from step to step for ``sequences`` sequences with the int8 caches ``kv`` (per layer ``kc/vc
    (B*heads, S, D)``, ``ks/vs (B*heads, S)``), or None when the model is not in the canonical form."""
    weights = read_weights(model) if _cabi.available() and model.model.embed_tokens.weight.dtype == torch.float16 else None
    if weights is None:
        return None
    size = int(_cabi.lib().lemoq_lockstep_workspace_bytes(describe(model, weights, max_len, kv)[0], sequences))
    if size == 0:
        return None
    workspace = torch.zeros(size, dtype=torch.uint8, device=model.model.embed_tokens.weight.device)
    return {"model": model, "kv": kv, "max_len": max_len, "workspace": workspace}


def run_lockstep(plan: dict, tokens: Any, position: Any, filled: Any, vocab: int, flags: Any) -> Any:
    """Logits ``(B, V)`` of one token per sequence; ``position`` and ``filled`` are device scalars.  None when the model has left the
    canonical form.  ``plan["weights"]``: the tensors this call reads (a captured step's graph reads them at every replay)."""
    weights = read_weights(plan["model"])
    if weights is None:
        return None
    desc, layers = describe(plan["model"], weights, plan["max_len"], plan["kv"])
    rows, workspace = int(tokens.shape[0]), plan["workspace"]
    logits = torch.empty((rows, vocab), dtype=torch.float16, device=tokens.device)
    _cabi.call("lemoq_lockstep_run", desc, layers, _cabi.ptr(tokens), _cabi.ptr(position), _cabi.ptr(filled), rows, _cabi.ptr(logits),
               _cabi.ptr(workspace), workspace.numel(), _cabi.ptr(flags), _cabi.current_stream(tokens.device))
    plan["weights"] = weights
    return logits
