"""Many tokens through the whole model in one native call, for models in the canonical W8 form: a prompt (``lemoq_prompt_run``), or one
token of each of many sequences (``lemoq_lockstep_run``).

The module tree's own forward stays the path of everything else; :func:`run_prompt`, :func:`lockstep_plan` and :func:`run_lockstep` return
None for what the native path does not take.  The model is read anew at every call, as its modules' forwards would read it: nothing of a
call is kept for the next by the address or identity of a tensor or module.
"""

from __future__ import annotations

from array import array
from itertools import chain, cycle
from typing import Any, NamedTuple

import torch
import torch.nn.functional as F
from torch import nn

from lemoq import _cabi, _native
from lemoq.kernels.attn_decode import _decode_forward_impl
from lemoq.kernels.moe_grouped_quant import QuantFusedExperts
from lemoq.kernels.rmsnorm import _fused_norm_forward
from lemoq.model import OlmoeAttention, OlmoeDecoderLayer, OlmoeRMSNorm, OlmoeRotaryEmbedding, StaticCache
from lemoq.quant.linear import QuantLinear

_PLAN = "_lemoq_prompt_plan"  # on the cache object: what the last native call over that cache was given

# the weights of a layer, in the order of ``LayerDesc``; behind them come the cache tensors
_LAYER_WEIGHTS = ("ln1", "ln2", "q_norm", "k_norm", "qkv_codes", "qkv_scale", "o_codes", "o_scale", "router", "gu_codes", "gu_scale", "dn_codes", "dn_scale")
_CACHES = ("keys", "values", "kc", "ks", "vc", "vs")
assert _LAYER_WEIGHTS + _CACHES == tuple(name for name, _ in _cabi.LayerDesc._fields_)


class Weights(NamedTuple):
    """The tensors of a model in the canonical form."""

    own: dict       # field of ``StepDesc`` -> tensor
    layers: list    # in the order of ``_LAYER_WEIGHTS``, layer after layer
    linears: list   # the W8 linears that a forward of the module tree calls
    unwatched: bool  # no hook on a module that such a forward calls, and none has another forward than the one computed natively

    def tensors(self) -> list:
        return [*self.own.values(), *self.layers]


_KNOWN = (OlmoeDecoderLayer, QuantLinear, QuantFusedExperts, OlmoeRMSNorm, _decode_forward_impl, OlmoeAttention.forward, F.silu, _fused_norm_forward, OlmoeRMSNorm.forward)
_NORM_FORWARDS = (_fused_norm_forward, OlmoeRMSNorm.forward)


def _plain(module: Any, forwards: tuple = ()) -> bool:
    """No hook, and no forward of its own but a bound method of one of ``forwards``."""
    own = module.__dict__.get("forward")
    return not (module._forward_hooks or module._forward_pre_hooks) and (own is None or getattr(own, "__func__", None) in forwards)


def _w8(linear: Any) -> tuple[Any, Any] | None:
    """Codes and scales of a W8 linear without bias that has them in the buffers it was built with, else None."""
    own = linear._buffers if type(linear) is QuantLinear else {}
    codes, scale = own.get("packed"), own.get("scale")
    return (codes, scale) if own.get("bias", linear) is None and codes is not None and scale is not None else None


def _read_layers(layers: list, group: int, eps: float, top_k: int, renormalised: bool) -> tuple[list, list, bool] | str:
    """(weights, linears, unwatched) of the decoder layers as ``Weights`` has them, or the reason why one description does not stand for them."""
    tensors, linears, unwatched = [], [], True
    for i, layer in enumerate(layers):
        if type(layer) is not OlmoeDecoderLayer:
            return "layer %d is a %s" % (i, type(layer).__name__)
        parts = layer._modules
        attn, mlp = parts["self_attn"], parts["mlp"]
        inner, here, moe = attn._modules, attn.__dict__, mlp.__dict__
        packed, o_proj, stacks = here.get("_lemoq_packed_qkv"), inner.get("o_proj"), moe.get("_static_experts")
        o_own = _w8(o_proj)
        if packed is None or o_own is None:
            return "layer %d: packed q/k/v not installed, or o_proj is not a W8 linear without bias" % i
        if not isinstance(stacks, QuantFusedExperts) or stacks.bits != 8 or moe["_static_act"] not in (None, F.silu):
            return "layer %d: experts are not W8 with SiLU" % i
        if (getattr(here.get("forward"), "__func__", None) is not _decode_forward_impl or here["num_key_value_groups"] != 1
                or getattr(here.get("_lemoq_original_forward"), "__func__", None) is not OlmoeAttention.forward):
            return "layer %d: attention core not replaced, or GQA" % i
        if not packed.group_size == o_proj.group_size == stacks.group_size == group:
            return ("layer %d: group sizes %d (q.k.v), %d (o_proj), %d (experts) beside %d (lm_head)"
                    % (i, packed.group_size, o_proj.group_size, stacks.group_size, group))
        if (moe["_static_top_k"], moe["_static_norm"]) != (top_k, renormalised):
            return "layer %d: top_k %d (normalised: %s) is not the configuration's" % (i, moe["_static_top_k"], moe["_static_norm"])
        norms = (parts["input_layernorm"], parts["post_attention_layernorm"], inner.get("q_norm"), inner.get("k_norm"))
        if any(type(norm) is not OlmoeRMSNorm or norm.variance_epsilon != eps or norm._parameters.get("weight") is None for norm in norms):
            return "layer %d: a norm is not RMSNorm with the configuration's eps" % i
        mine = [o_proj, *filter(None, map(inner.get, ("q_proj", "k_proj", "v_proj")))]  # (absent where only the stacked rows were kept)
        block_forward = getattr(moe.get("forward"), "of_block", None) is mlp and not (mlp._forward_hooks or mlp._forward_pre_hooks)
        unwatched = (unwatched and block_forward and _plain(layer) and _plain(attn, (_decode_forward_impl,)) and all(_plain(n, _NORM_FORWARDS) for n in norms)
                     and all(type(x) is QuantLinear and _plain(x) for x in mine))
        linears += mine
        tensors += [*(norm._parameters["weight"] for norm in norms), packed.packed, packed.scale, *o_own,
                    moe["_static_router"].contiguous(), stacks.packed_gate_up, stacks.scale_gate_up, stacks.packed_down, stacks.scale_down]
    return tensors, linears, unwatched


def _read(model: Any) -> tuple[Weights | None, str | None]:
    """The tensors that the model's forwards would use now, or None and the reason why one ``StepDesc`` does not stand for the model: it has
    ONE group size, top_k, eps and so on, so what every block was really built with is compared here."""
    cfg, m, lm = model.config, model._modules["model"], model._modules["lm_head"]
    parts = m._modules
    embed, norm, rotary, layers = parts["embed_tokens"], parts["norm"], parts["rotary_emb"], list(parts["layers"]._modules.values())
    lm_own = _w8(lm)
    if lm_own is None:
        return None, "lm_head is not a W8 linear without bias"
    if cfg.clip_qkv is not None or not layers:
        return None, "clip_qkv is set, or there are no layers"
    if type(norm) is not OlmoeRMSNorm or norm.variance_epsilon != cfg.rms_norm_eps or embed._parameters.get("weight") is None or norm._parameters.get("weight") is None:
        return None, "the embedding or the final norm is not the configuration's"
    wanted = (lm.group_size, cfg.rms_norm_eps, cfg.num_experts_per_tok, bool(cfg.norm_topk_prob))
    found = _native.layers(layers, _KNOWN, wanted) or _read_layers(layers, *wanted)
    if isinstance(found, str):
        return None, found
    tensors, linears, unwatched = found
    unwatched = (unwatched and type(embed) is nn.Embedding and embed.max_norm is None and type(rotary) is OlmoeRotaryEmbedding
                 and _plain(lm) and _plain(embed) and _plain(rotary) and _plain(norm, _NORM_FORWARDS))
    own = {"embed": embed._parameters["weight"], "final_norm": norm._parameters["weight"], "lm_head_codes": lm_own[0], "lm_head_scale": lm_own[1]}
    return Weights(own, tensors, [lm, *linears], unwatched), None


def read_weights(model: Any) -> Weights | None:
    return _read(model)[0]


def _skippable(weights: Weights) -> bool:
    """May the module tree's forward be left out?  Not when that would be noticed."""
    every = torch.nn.modules.module
    return weights.unwatched and not (every._global_forward_hooks or every._global_forward_pre_hooks)


_HALF, _CODE = 0, 1  # element types of a form: (type, *shape)


def _forms(model: Any) -> tuple[tuple, tuple]:
    """What the C side takes the model's own tensors and those of a layer to be: it computes every offset from the sizes alone."""
    cfg, g = model.config, int(model.lm_head.group_size)
    h, a, f, e, v = cfg.hidden_size, cfg.num_attention_heads * cfg.head_dim, cfg.intermediate_size, cfg.num_experts, cfg.vocab_size
    own = ((_HALF, v, h), (_HALF, h), (_CODE, v, h), (_HALF, v, h // g))
    return own, ((_HALF, h), (_HALF, h), (_HALF, a), (_HALF, a), (_CODE, 3 * a, h), (_HALF, 3 * a, h // g), (_CODE, h, a), (_HALF, h, a // g), (_HALF, e, h),
                 (_CODE, e, 2 * f, h), (_HALF, e, 2 * f, h // g), (_CODE, e, h, f), (_HALF, e, h, f // g))


def _misfit(tensors: list, forms: tuple, names: tuple, device: Any) -> str | None:
    """The first tensor that is not contiguous, 16-byte aligned, on ``device`` and of its form."""
    for i, t in enumerate(tensors):
        form, name = forms[i % len(forms)], names[i % len(names)]
        if t.dtype is not (torch.float16, torch.int8)[form[0]] or tuple(t.shape) != form[1:] or t.device != device:
            return "%s is %s %s on %s" % (name, tuple(t.shape), t.dtype, t.device)
        if not t.is_contiguous() or t.data_ptr() & 15:
            return "%s is not contiguous and 16-byte aligned" % name
    return None


def _pointers(tensors: list, forms: tuple, names: tuple, device: Any, caches: list = [], cache_forms: tuple = ()) -> bytes | None:  # noqa: B006
    """The tensors' addresses, 64 bits each, behind the weights of every layer those of its caches (None: 0); None when one of them misfits."""
    index = -1 if device.index is None else device.index
    words = _native.pointers(tensors, forms, index, caches, cache_forms) if caches else _native.pointers(tensors, forms, index)
    if words is not None:
        return words
    there = [(t, form, name) for t, form, name in zip(caches, cycle(cache_forms), cycle(_CACHES)) if t is not None]
    if _misfit(tensors, forms, names, device) or any(_misfit([t], (form,), (name,), device) for t, form, name in there):
        return None
    address = lambda t: 0 if t is None else t.data_ptr()  # noqa: E731
    w, c = len(forms), len(cache_forms)
    rounds = [[*map(address, tensors[r * w: (r + 1) * w]), *map(address, caches[r * c: (r + 1) * c])] for r in range(len(tensors) // w)]
    return array("Q", chain.from_iterable(rounds)).tobytes()


def form_blocker(model: Any) -> str | None:
    """Why the native paths' one set of sizes does not describe the model (None: it does)."""
    weights, reason = _read(model)
    if weights is None:
        return reason
    if any(n % model.lm_head.group_size for n in (model.config.hidden_size, model.config.intermediate_size)):
        return "group size %d does not divide every row" % model.lm_head.group_size
    own, layer = _forms(model)
    device = weights.own["embed"].device
    return (_misfit(list(weights.own.values()), own, tuple(weights.own), device)
            or _misfit(weights.layers, layer, _LAYER_WEIGHTS, device))


def describe(model: Any, weights: Weights, max_len: int, caches: list[tuple], cache_forms: tuple) -> tuple[Any, Any] | None:
    """``(StepDesc, LayerDesc array)`` of the model over one set of cache tensors per layer (in the order of ``_CACHES``, each None or of its form):
    pointers only, the caller keeps the tensors for as long as the C side may read them.  None when a tensor misfits."""
    cfg, device, (own_forms, layer_forms) = model.config, weights.own["embed"].device, _forms(model)
    own = _pointers(list(weights.own.values()), own_forms, tuple(weights.own), device)
    words = _pointers(weights.layers, layer_forms, _LAYER_WEIGHTS, device, list(chain.from_iterable(caches)), cache_forms)
    if own is None or words is None:
        return None
    cos, sin = model.model.rotary_emb.tables(max_len, torch.float16, device)
    desc = _cabi.StepDesc(len(caches), cfg.hidden_size, cfg.num_attention_heads, cfg.head_dim, cfg.num_experts, cfg.num_experts_per_tok, cfg.intermediate_size,
                          cfg.vocab_size, int(model.lm_head.group_size), max_len, float(cfg.rms_norm_eps), int(bool(cfg.norm_topk_prob)), 0, 0, 0,
                          *array("Q", own), cos.data_ptr(), sin.data_ptr())
    return desc, (_cabi.LayerDesc * len(caches)).from_buffer_copy(words)


def _operations_matter() -> bool:
    """Is somebody to see or change the single operations of this call (autocast, a dispatch mode, a trace, a compilation)?"""
    return bool(torch.compiler.is_compiling() or torch.is_autocast_enabled("cuda") or torch._C._len_torch_dispatch_stack() or torch.jit.is_tracing())


def run_prompt(model: Any, input_ids: Any, cache: Any, cache_position: Any, position_ids: Any) -> Any:
    """Logits ``(1, T, V)`` of the prompt ``input_ids (1, T)``, with its K/V rows written into ``cache`` - or None when the
    model, the cache or the call is not of the kind the native path takes.  A token id outside the vocabulary, a position outside the cache
    and a wait that ran out raise ``RuntimeError`` (the kernels clamp and flag; the call waits for the flag unless the cache's owner does)."""

    if _operations_matter():
        return None
    weight = model.model.embed_tokens.weight
    if (torch.is_grad_enabled() or type(cache) is not StaticCache or input_ids.shape[0] != 1 or not weight.is_cuda or weight.dtype != torch.float16
            or input_ids.dtype != torch.int64 or cache_position.dtype != torch.int64 or not cache_position.is_cuda or cache_position.numel() != input_ids.shape[1]
            or position_ids.data_ptr() != cache_position.data_ptr() or position_ids.numel() != cache_position.numel() or not cache_position.is_contiguous()
            or len(cache.layers) != len(model.model.layers) or not _cabi.available()):
        return None
    weights = read_weights(model)
    if weights is None or not _skippable(weights):
        return None
    cfg, device = model.config, weight.device
    for slot in cache.layers:
        if not slot.is_initialized:
            slot.lazy_initialization(torch.empty((1, cfg.num_attention_heads, 1, cfg.head_dim), dtype=torch.float16, device=device))
    described = describe(model, weights, cache.max_cache_len, [(s.keys, s.values, None, None, None, None) for s in cache.layers],
                         6 * ((_HALF, 1, cfg.num_attention_heads, cache.max_cache_len, cfg.head_dim),))
    if described is None:
        return None
    desc, layers = described
    tokens = int(input_ids.shape[1])
    size = int(_cabi.lib().lemoq_prompt_workspace_bytes(desc, tokens))
    if size == 0:
        return None
    # the error word: the one the cache carries, whose owner reads it, or one of this call's own
    carried = cache.__dict__.get("_lemoq_error_word")
    flags = torch.zeros(1, dtype=torch.int32, device=device) if carried is None else carried
    cache.__dict__[_PLAN] = {"flags": flags}
    ids = input_ids.contiguous()
    logits = torch.empty((1, tokens, cfg.vocab_size), dtype=torch.float16, device=device)
    workspace = torch.empty(size, dtype=torch.uint8, device=device)
    _cabi.call("lemoq_prompt_run", desc, layers, _cabi.ptr(ids), _cabi.ptr(cache_position), tokens, _cabi.ptr(logits),
               _cabi.ptr(workspace), size, _cabi.ptr(flags), _cabi.current_stream(device))
    for linear in weights.linears:
        linear.count_separate(several=True)
    if carried is None and not torch.cuda.is_current_stream_capturing():
        _cabi.check_flags(int(flags), "prompt")
    return logits


def _describe_lockstep(model: Any, weights: Weights, kv: list[dict], sequences: int, max_len: int) -> tuple[Any, Any] | None:
    heads, dim = sequences * model.config.num_attention_heads, model.config.head_dim
    codes, scales = (_CODE, heads, max_len, dim), (_HALF, heads, max_len)
    return describe(model, weights, max_len, [tuple(map(slots.get, _CACHES)) for slots in kv], (codes, codes, codes, scales, codes, scales))


def lockstep_plan(model: Any, kv: list[dict], sequences: int, max_len: int) -> dict | None:
    """What :func:`run_lockstep` keeps from step to step for ``sequences`` sequences with the int8 caches ``kv`` (per layer ``kc/vc
    (B*heads, S, D)``, ``ks/vs (B*heads, S)``), or None when the model is not in the canonical form."""
    weights = read_weights(model) if _cabi.available() else None
    described = None if weights is None else _describe_lockstep(model, weights, kv, sequences, max_len)
    if described is None:
        return None
    size = int(_cabi.lib().lemoq_lockstep_workspace_bytes(described[0], sequences))
    if size == 0:
        return None
    workspace = torch.zeros(size, dtype=torch.uint8, device=model.model.embed_tokens.weight.device)
    return {"model": model, "kv": kv, "max_len": max_len, "workspace": workspace, "sequences": sequences}


def run_lockstep(plan: dict, tokens: Any, position: Any, filled: Any, vocab: int, flags: Any) -> Any:
    """Logits ``(B, V)`` of one token per sequence; ``position`` and ``filled`` are device scalars.  None when the model has left the
    canonical form.  ``plan["weights"]``: the tensors this call reads (a captured step's graph reads them at every replay)."""
    model, max_len = plan["model"], plan["max_len"]
    weights = read_weights(model)
    described = None if weights is None else _describe_lockstep(model, weights, plan["kv"], plan["sequences"], max_len)
    if described is None:
        return None
    desc, layers = described
    rows, workspace = int(tokens.shape[0]), plan["workspace"]
    logits = torch.empty((rows, vocab), dtype=torch.float16, device=tokens.device)
    _cabi.call("lemoq_lockstep_run", desc, layers, _cabi.ptr(tokens), _cabi.ptr(position), _cabi.ptr(filled), rows, _cabi.ptr(logits),
               _cabi.ptr(workspace), workspace.numel(), _cabi.ptr(flags), _cabi.current_stream(tokens.device))
    plan["weights"] = weights
    return logits
