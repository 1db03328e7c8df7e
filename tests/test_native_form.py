"""How the native paths read a model (no GPU), and which they leave to the module tree."""

from __future__ import annotations

import os

import pytest
import torch

from oracle import lemoq_oracle as ops


@pytest.fixture(params=["binding", "python"])
def canonical(request, monkeypatch):
    """Builder of a small canonical model on the CPU; ``experts``: group size of the experts' scales.  Everything is asked of the binding's
    functions and of the Python expressions they stand for."""
    from lemoq import _native
    import lemoq.quant.rtn as rtn
    from lemoq.kernels.attn_decode import replace_attention_cores
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts
    from lemoq.kernels.moe_static import fuse_experts, replace_moe_blocks
    from lemoq.kernels.packed_qkv import install_packed_qkv
    from lemoq.kernels.rmsnorm import replace_rms_norms
    from lemoq.model import OlmoeConfig, OlmoeForCausalLM
    from lemoq.quant.linear import SchemeSpec, quantize_model

    monkeypatch.setattr(rtn, "quantize_w8", lambda w, g=128: ops.rtn_quantize_w8(w.detach().float(), g))

    def build(experts=128):
        torch.manual_seed(0)
        cfg = OlmoeConfig(vocab_size=64, hidden_size=256, intermediate_size=256, num_hidden_layers=2, num_attention_heads=2,
                          num_key_value_heads=2, num_experts=8, num_experts_per_tok=2)
        model = OlmoeForCausalLM(cfg).to(torch.float16).eval()
        packed = {}
        for i, layer in enumerate(model.model.layers):
            fused = fuse_experts(layer.mlp.experts)
            packed[i] = QuantFusedExperts(*ops.rtn_quantize_w8(fused.gate_up.float(), experts), *ops.rtn_quantize_w8(fused.down.float(), experts), 8, experts)
        replace_rms_norms(model, "fused")
        replace_moe_blocks(model, impl="grouped", prequantized=packed)
        quantize_model(model, SchemeSpec.from_flags("w8a16", 128, targets=("attention", "experts", "lm_head"), keep_lm_head_fp16=False))
        replace_attention_cores(model, backend="cuda")
        install_packed_qkv(model)
        return model

    if request.param == "python":
        for name in ("layers", "pointers"):
            monkeypatch.setattr(_native, name, lambda *a: None)
    else:  # an ordinary model is the binding's business: nothing of it is asked of the Python expressions
        from lemoq import prompt

        model = build()
        with monkeypatch.context() as patch:
            patch.setattr(prompt, "_read_layers", None)
            patch.setattr(prompt, "_misfit", None)
            assert prompt._skippable(prompt.read_weights(model))
            assert prompt.describe(model, prompt.read_weights(model), 8, 2 * [6 * (None,)], 6 * ((prompt._HALF,),)) is not None
    return build


def test_a_description_follows_the_tensors_of_the_model(canonical):
    """Nothing is kept by a module's identity: whatever replaces a parameter or a buffer is what the next call is given."""
    from lemoq.prompt import _HALF, describe, read_weights

    model, forms = canonical(), 6 * ((_HALF, 1, 2, 8, 128),)
    caches = [(torch.zeros(1, 2, 8, 128, dtype=torch.float16), torch.zeros(1, 2, 8, 128, dtype=torch.float16), *4 * (None,)) for _ in range(2)]

    def pointers():
        desc, layers = describe(model, read_weights(model), 8, caches, forms)
        return [getattr(desc, n) for n in ("embed", "final_norm", "lm_head_codes", "lm_head_scale")], [[getattr(d, n) for n, _ in d._fields_] for d in layers]

    def moved():
        """Fields of the model and of the last layer that are given other tensors than before."""
        nonlocal before
        after = pointers()
        names = [n for n, a, b in zip(("embed", "final_norm", "lm_head_codes", "lm_head_scale"), before[0], after[0]) if a != b]
        names += [n for (n, _), a, b in zip(type(describe(model, read_weights(model), 8, caches, forms)[1][0])._fields_, before[1][-1], after[1][-1]) if a != b]
        before = after
        return names

    before, last = pointers(), model.model.layers[-1]
    keep = []  # nothing may land where the old tensor was
    for change, expected in ((lambda: setattr(last.input_layernorm, "weight", torch.nn.Parameter(last.input_layernorm.weight.clone())), ["ln1"]),
                             (lambda: setattr(last.self_attn.q_norm.weight, "data", last.self_attn.q_norm.weight.data.clone()), ["q_norm"]),
                             (lambda: setattr(last.self_attn.o_proj, "packed", last.self_attn.o_proj.packed.clone()), ["o_codes"]),
                             (lambda: setattr(last.mlp._static_experts, "scale_down", last.mlp._static_experts.scale_down.clone()), ["dn_scale"]),
                             (lambda: model.lm_head.load_state_dict({k: v.clone() for k, v in model.lm_head.state_dict().items()}, assign=True),
                              ["lm_head_codes", "lm_head_scale"]),
                             (lambda: caches.append((caches.pop()[0].clone(), *caches[0][1:])), ["keys", "values"])):
        keep.append([t.detach() for t in read_weights(model).tensors()] + [t for c in caches for t in c[:2]])
        change()
        assert moved() == expected
    last.self_attn.o_proj.bias = torch.zeros(256)
    assert read_weights(model) is None  # and what it no longer describes is not taken


@pytest.mark.parametrize("group", [64, 256])
def test_experts_of_another_group_size_are_not_one_description(canonical, group):
    from lemoq.prompt import form_blocker

    assert form_blocker(canonical()) is None
    assert "group sizes 128 (q.k.v), 128 (o_proj), %d (experts) beside 128" % group in form_blocker(canonical(experts=group))


def test_every_block_is_compared_with_the_configuration(canonical):
    from lemoq.prompt import form_blocker

    model = canonical()
    first, last = model.model.layers
    for owner, name, value, told in ((last.mlp, "_static_top_k", 3, "top_k 3"), (last.mlp, "_static_norm", True, "normalised: True"),
                                     (first.mlp, "_static_act", torch.relu, "SiLU"), (last.self_attn.q_norm, "variance_epsilon", 1e-6, "eps"),
                                     (model.lm_head, "bias", torch.zeros(64), "bias"), (first.self_attn.o_proj, "bias", torch.zeros(256), "bias"),
                                     (first.mlp, "_static_router", first.mlp._static_router[:4], "router"),
                                     (last.self_attn._lemoq_packed_qkv, "scale", last.self_attn._lemoq_packed_qkv.scale.float(), "qkv_scale"),
                                     (last.mlp._static_experts, "scale_down", torch.zeros(8 * 256 * 2 + 1, dtype=torch.float16)[1:].view(8, 256, 2), "aligned")):
        kept = getattr(owner, name)
        setattr(owner, name, value)
        assert told in form_blocker(model), name
        setattr(owner, name, kept)
    assert form_blocker(model) is None


def test_a_tensor_of_another_form_is_not_described(canonical):
    from lemoq.prompt import _HALF, describe, read_weights

    model, forms = canonical(), 6 * ((_HALF, 1, 2, 8, 128),)
    cache = lambda n: [(torch.zeros(1, 2, n, 128, dtype=torch.float16), torch.zeros(1, 2, 8, 128, dtype=torch.float16), *4 * (None,)) for _ in range(2)]  # noqa: E731
    assert describe(model, read_weights(model), 8, cache(8), forms) is not None and describe(model, read_weights(model), 8, cache(9), forms) is None
    mlp = model.model.layers[1].mlp
    whole = mlp._static_experts.packed_down
    for other in (whole[:7], whole.to(torch.int16), whole.to("meta"), whole.transpose(1, 2).contiguous().transpose(1, 2),
                  torch.zeros(whole.numel() + 1, dtype=torch.int8)[1:].view_as(whole)):
        mlp._static_experts.packed_down = other
        assert describe(model, read_weights(model), 8, cache(8), forms) is None


def test_a_forward_that_is_seen_or_replaced_is_not_skipped(canonical):
    from lemoq.prompt import _skippable, read_weights

    model = canonical()
    layer = model.model.layers[1]
    skippable = lambda: (lambda weights: weights is not None and _skippable(weights))(read_weights(model))  # noqa: E731
    assert skippable() and len(read_weights(model).linears) == 9
    called = [model.lm_head, model.model.norm, model.model.embed_tokens, model.model.rotary_emb, layer, layer.self_attn, layer.mlp, layer.input_layernorm,
              *(getattr(layer.self_attn, n) for n in ("q_proj", "k_proj", "v_proj", "o_proj", "q_norm", "k_norm")), layer.post_attention_layernorm]
    for module in called:
        for register in (module.register_forward_hook, module.register_forward_pre_hook):
            handle = register(lambda *a: None)
            assert not skippable(), module
            handle.remove()
        own = module.__dict__.get("forward")
        module.forward = lambda *a, **k: None
        assert not skippable(), module
        del module.forward
        if own is not None:
            module.forward = own
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert not skippable()
    handle.remove()
    assert skippable()


def test_projections_may_be_given_up_once_they_are_stacked(canonical):
    from lemoq.prompt import _skippable, form_blocker, read_weights

    model = canonical()
    for layer in model.model.layers:
        del layer.self_attn.q_proj, layer.self_attn.k_proj, layer.self_attn.v_proj
    assert form_blocker(model) is None and _skippable(read_weights(model))


def test_a_router_of_other_strides_is_laid_out(canonical):
    from lemoq.prompt import form_blocker, read_weights

    model = canonical()
    mlp = model.model.layers[1].mlp
    mlp._static_router = mlp._static_router.t().contiguous().t()
    assert form_blocker(model) is None and torch.equal(read_weights(model).layers[13 + 8], mlp._static_router)


@pytest.mark.parametrize("name", ["bias", "scale", "packed"])
def test_a_linear_whose_tensors_are_no_buffers_goes_through_the_modules(canonical, name):
    from lemoq.prompt import form_blocker, read_weights

    model = canonical()
    for linear in (model.lm_head, model.model.layers[1].self_attn.o_proj):
        kept = getattr(linear, name)
        setattr(linear, name, torch.nn.Parameter(torch.ones(64) if kept is None else kept.clone(), requires_grad=False))
        assert read_weights(model) is None and "not a W8 linear without bias" in form_blocker(model)
        delattr(linear, name)
        linear.register_buffer(name, kept)
    assert form_blocker(model) is None


@pytest.mark.parametrize("tokens", [1, 3])
@pytest.mark.parametrize("mode", ["fused", "separate"])
@pytest.mark.parametrize("name", ["bias", "scale"])
@pytest.mark.parametrize("kind", ["assigned", "parametrised"])
def test_a_tensor_of_a_quant_linear_need_not_be_a_buffer(monkeypatch, kind, name, mode, tokens):
    """A bias or scale assigned as a parameter (for tuning), or parametrised, is what the linear computes with, and its gradient is there."""
    import lemoq.quant.rtn as rtn
    from lemoq.quant.linear import QuantLinear, SchemeSpec

    monkeypatch.setattr(rtn, "quantize_w8", lambda w, g=128: ops.rtn_quantize_w8(w.detach().float(), g))
    torch.manual_seed(tokens)
    linear = QuantLinear(torch.nn.Linear(128, 64), SchemeSpec.from_flags("w8a16", 128, dequant=mode))
    codes, tensors = linear.packed.float(), {"scale": linear.scale.float(), "bias": linear.bias.float()}
    if kind == "assigned":
        setattr(linear, name, torch.nn.Parameter(2 * tensors[name]))
    else:
        class Twice(torch.nn.Module):
            def forward(self, t):
                return 2 * t.float()

        torch.nn.utils.parametrize.register_parametrization(linear, name, Twice(), unsafe=True)
    tensors[name] = 2 * tensors[name]
    x = torch.randn(tokens, 128)
    got = linear(x)
    # fp32 throughout, the same weight: sums of 128 products in another order, 128 x 2^-24
    assert torch.allclose(got, x @ (codes * tensors["scale"]).t() + tensors["bias"], rtol=1e-5, atol=1e-5)
    if kind == "assigned":
        got.sum().backward()
        assert getattr(linear, name).grad.abs().sum() > 0


def test_an_expert_tile_waits_for_every_word_it_reads(tmp_path):
    """The routing words of the whole-step kernel may become visible in any order: whatever words have come, a tile is taken up only when each of
    its own carries the layer's mark, and the tiles of a layer hold every slot once."""
    import ctypes
    import subprocess

    from conftest import PKG

    source, lib = tmp_path / "route.cpp", tmp_path / "route.so"
    source.write_text("""#include "step_route.h"
    using namespace lemoq::tile;
    extern "C" int slots(int down, int tile, int shift, int paired, int top_k, int* count) {
        const RouteSlots s = down ? slots_of_down(tile, paired, top_k) : slots_of_gate_up(tile, shift);
        *count = s.count;
        return s.first;
    }
    extern "C" int known(const uint32_t* route, int layer, int first, int count) { return route_known(route, layer, RouteSlots{first, count}); }
    extern "C" uint32_t word(int layer, int expert) { return route_mark(layer) | static_cast<uint32_t>(expert); }
    extern "C" uint32_t expert(uint32_t word) { return route_expert(word); }
    """)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), str(source), "-o", str(lib)], check=True)
    native, layer = ctypes.CDLL(str(lib)), 31
    assert native.expert(native.word(layer, 127)) == 127
    for down, paired, top_k in [(0, 0, 4), *((1, p, k) for p in (0, 1) for k in (1, 2, 5, 8))]:
        tiles = 4 * top_k if not down else -(-top_k // 2) if paired else top_k
        held = []
        for tile in range(tiles):
            count = ctypes.c_int()
            first = native.slots(down, tile, 2, paired, top_k, ctypes.byref(count))
            own = set(range(first, first + count.value))
            held += own
            for come in range(1 << top_k):  # the words of this layer that can be seen; the others still hold the layer before's
                words = [native.word(layer if come >> k & 1 else layer - 1, k) for k in range(top_k)]
                ready = native.known((ctypes.c_uint32 * 32)(*words), layer, first, count.value)
                assert bool(ready) == all(come >> k & 1 for k in own), (down, paired, top_k, tile, come)
        assert sorted(held) == sorted(list(range(top_k)) * (1 if down else 4))
