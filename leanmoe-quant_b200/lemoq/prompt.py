"""Many tokens through the whole model in one native call, for models in the canonical W8 form: a prompt (``lemoq_prompt_run``), or one
token of each of many sequences (``lemoq_lockstep_run``).

The module tree's own forward stays the path of everything else; :func:`run_prompt` and :func:`lockstep_plan` return None for
what the native path does not take.
"""

from __future__ import annotations

from typing import Any

import torch
import torch.nn.functional as F

from lemoq import _cabi

_PLAN = "_lemoq_prompt_plan"  # on the cache object: descriptors of one model over that cache


def _layer_parts(layer: Any) -> tuple | None:
    """The quantised pieces of a decoder layer, or None when a piece is not in the form the native path knows."""
    from lemoq.kernels.attn_decode import _decode_forward_impl
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts
    from lemoq.model import OlmoeAttention
    from lemoq.quant.linear import QuantLinear

    attn, mlp = layer.self_attn, layer.mlp
    here = attn.__dict__
    packed, o_proj = here.get("_lemoq_packed_qkv"), attn.o_proj
    stacks = mlp.__dict__.get("_static_experts")
    plain = getattr(here.get("_lemoq_original_forward"), "__func__", None)
    ok = (packed is not None and isinstance(o_proj, QuantLinear) and o_proj.bias is None and isinstance(stacks, QuantFusedExperts)
          and getattr(here.get("forward"), "__func__", None) is _decode_forward_impl and plain is OlmoeAttention.forward
          and attn.num_key_value_groups == 1 and mlp._static_act in (None, F.silu))
    return (attn, mlp, packed, o_proj, stacks) if ok else None


def _signature(model: Any) -> tuple | None:
    """The objects a plan was made from; None when the model is not in the canonical form."""
    from lemoq.quant.linear import QuantLinear

    cfg, lm = model.config, model.lm_head
    if not isinstance(lm, QuantLinear) or lm.bias is not None or cfg.clip_qkv is not None:
        return None
    parts = [_layer_parts(layer) for layer in model.model.layers]
    if not parts or any(p is None for p in parts):
        return None
    return (lm, model.model.embed_tokens.weight, *parts)


def _describe(model: Any, signature: tuple, max_len: int, caches: list[dict]) -> dict:
    """The model and one set of cache tensors per layer (named as in ``LayerDesc``) for the C side: pointers only."""
    cfg, m = model.config, model.model
    device = m.embed_tokens.weight.device
    cos, sin = m.rotary_emb.tables(max_len, torch.float16, device)
    layers = (_cabi.LayerDesc * len(m.layers))()
    keep: list[Any] = [cos, sin]
    for d, layer, (attn, mlp, packed, o_proj, stacks), slots in zip(layers, m.layers, signature[2:], caches):
        router = mlp._static_router.contiguous()
        keep += [router, slots]
        tensors = {"ln1": layer.input_layernorm.weight, "ln2": layer.post_attention_layernorm.weight, "q_norm": attn.q_norm.weight,
                   "k_norm": attn.k_norm.weight, "qkv_codes": packed.packed, "qkv_scale": packed.scale, "o_codes": o_proj.packed,
                   "o_scale": o_proj.scale, "router": router, "gu_codes": stacks.packed_gate_up, "gu_scale": stacks.scale_gate_up,
                   "dn_codes": stacks.packed_down, "dn_scale": stacks.scale_down, **slots}
        for name, t in tensors.items():
            setattr(d, name, _cabi.ptr(t))
    desc = _cabi.StepDesc()
    desc.layers, desc.hidden, desc.heads, desc.head_dim = len(m.layers), cfg.hidden_size, cfg.num_attention_heads, cfg.head_dim
    desc.experts, desc.top_k, desc.ffn, desc.vocab = cfg.num_experts, cfg.num_experts_per_tok, cfg.intermediate_size, cfg.vocab_size
    desc.group_size, desc.max_len, desc.eps = int(model.lm_head.group_size), max_len, float(cfg.rms_norm_eps)
    desc.norm_topk_prob = int(bool(cfg.norm_topk_prob))
    desc.embed, desc.final_norm = _cabi.ptr(m.embed_tokens.weight), _cabi.ptr(m.norm.weight)
    desc.lm_head_codes, desc.lm_head_scale = _cabi.ptr(model.lm_head.packed), _cabi.ptr(model.lm_head.scale)
    desc.rope_cos, desc.rope_sin = _cabi.ptr(cos), _cabi.ptr(sin)
    return {"signature": signature, "desc": desc, "layers": layers, "keep": keep}


def _prompt_plan(model: Any, cache: Any, signature: tuple) -> dict:
    cfg, device = model.config, model.model.embed_tokens.weight.device
    for slot in cache.layers:
        if not slot.is_initialized:
            slot.lazy_initialization(torch.empty((1, cfg.num_attention_heads, 1, cfg.head_dim), dtype=torch.float16, device=device))
    plan = _describe(model, signature, cache.max_cache_len, [{"keys": s.keys, "values": s.values} for s in cache.layers])
    plan.update(caches=tuple(s.keys for s in cache.layers), flags=torch.zeros(1, dtype=torch.int32, device=device))
    return plan


def _same(a: tuple, b: tuple) -> bool:
    return len(a) == len(b) and all(x is y or (isinstance(x, tuple) and _same(x, y)) for x, y in zip(a, b))


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
    signature = _signature(model)
    if signature is None:
        return None
    plan = cache.__dict__.get(_PLAN)
    if plan is None or not _same(plan["signature"], signature) or any(s.keys is not k for s, k in zip(cache.layers, plan["caches"])):
        plan = cache.__dict__[_PLAN] = _prompt_plan(model, cache, signature)
    tokens = int(input_ids.shape[1])
    size = int(_cabi.lib().lemoq_prompt_workspace_bytes(plan["desc"], tokens))
    if size == 0:
        return None
    ids, device = input_ids.contiguous(), weight.device
    logits = torch.empty((1, tokens, model.config.vocab_size), dtype=torch.float16, device=device)
    workspace = torch.empty(size, dtype=torch.uint8, device=device)
    _cabi.call("lemoq_prompt_run", plan["desc"], plan["layers"], _cabi.ptr(ids), _cabi.ptr(cache_position), tokens, _cabi.ptr(logits),
               _cabi.ptr(workspace), size, _cabi.ptr(plan["flags"]), _cabi.current_stream(device))
    return logits


def lockstep_plan(model: Any, kv: list[dict], sequences: int, max_len: int) -> Any:
    """What :func:`run_lockstep` needs for ``sequences`` sequences with the int8 caches ``kv`` (per layer ``kc/vc (B*heads, S, D)``,
    ``ks/vs (B*heads, S)``), or None when the model is not in the canonical form."""
    signature = _signature(model) if _cabi.available() and model.model.embed_tokens.weight.dtype == torch.float16 else None
    if signature is None:
        return None
    plan = _describe(model, signature, max_len, kv)
    size = int(_cabi.lib().lemoq_lockstep_workspace_bytes(plan["desc"], sequences))
    if size == 0:
        return None
    plan["workspace"] = torch.zeros(size, dtype=torch.uint8, device=model.model.embed_tokens.weight.device)
    return plan


def run_lockstep(plan: dict, tokens: Any, position: Any, filled: Any, vocab: int, flags: Any) -> Any:
    """Logits ``(B, V)`` of one token per sequence; ``position`` and ``filled`` are device scalars."""
    rows, workspace = int(tokens.shape[0]), plan["workspace"]
    logits = torch.empty((rows, vocab), dtype=torch.float16, device=tokens.device)
    _cabi.call("lemoq_lockstep_run", plan["desc"], plan["layers"], _cabi.ptr(tokens), _cabi.ptr(position), _cabi.ptr(filled), rows, _cabi.ptr(logits),
               _cabi.ptr(workspace), workspace.numel(), _cabi.ptr(flags), _cabi.current_stream(tokens.device))
    return logits
