"""The tensor-core kernels for many tokens at the edges of their tiles, and a whole prompt through ``lemoq_prompt_run``, against the CPU
oracle."""

from __future__ import annotations

import pytest
import torch

from gpu_util import PER_KERNEL_REL_TOL, install_canonical, lemoq_model_from_oracle, rel_err
from oracle import lemoq_oracle as ops
from oracle import olmoe_decode_oracle as glue

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _w8(n, k, seed, experts=0):
    w = torch.randn(*((experts,) if experts else ()), n, k, generator=torch.Generator().manual_seed(seed)) * 0.02
    return ops.rtn_quantize_w8(w, 128)


def _gemm(x, codes, scale, *, seg=None, gate_up=False, exact=True, resid=None):
    from lemoq import _cabi

    n, k = codes.shape[-2:]
    y = torch.full((x.shape[0], n // 2 if gate_up else n), float("nan"), dtype=torch.float16, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    _cabi.call("lemoq_w8_gemm", _cabi.ptr(x), x.shape[0], _cabi.ptr(codes), _cabi.ptr(scale), n, k, 128, _cabi.ptr(seg),
               codes.shape[0] if codes.dim() == 3 else 1, int(gate_up), int(exact), _cabi.ptr(resid), _cabi.ptr(y), _cabi.ptr(flag), _cabi.current_stream())
    assert int(flag) == 0
    return y


# one token; either side of the 16-, 32-, 64- and 128-token tiles; rows that leave a tile of 256 half empty or spill over it; one
# group of codes, and an odd number of them
@pytest.mark.parametrize("tokens,n,k,exact", [(1, 2, 128, True), (16, 256, 128, True), (17, 130, 384, True), (33, 258, 256, True), (64, 514, 640, True),
                                              (65, 256, 128, True), (65, 258, 384, False), (128, 128, 256, False), (129, 770, 128, False), (300, 256, 640, False),
                                              # groups shared out over a cluster: evenly, unevenly, more parts than tokens
                                              (64, 514, 2048, True), (33, 2048, 1152, True), (3, 130, 1024, True)])
def test_w8_gemm_edges(tokens, n, k, exact):
    codes, scale = _w8(n, k, tokens + n)
    x = torch.randn(tokens, k, generator=torch.Generator().manual_seed(k)).half()
    resid = torch.randn(tokens, n, generator=torch.Generator().manual_seed(n)).half()
    ref = ops.dense_w8_gemv(x, codes, scale, 128)
    args = (x.to(DEV), codes.to(DEV), scale.to(DEV))
    assert rel_err(_gemm(*args, exact=exact), ref) < PER_KERNEL_REL_TOL
    assert rel_err(_gemm(*args, exact=exact, resid=resid.to(DEV)), ref.half() + resid) < PER_KERNEL_REL_TOL
    gate, up = ref.float()[:, : n // 2], ref.float()[:, n // 2:]
    assert rel_err(_gemm(*args, exact=exact, gate_up=True), gate * torch.sigmoid(gate) * up) < 2 * PER_KERNEL_REL_TOL


@pytest.mark.parametrize("tokens", [3, 70, 130])  # exact form; scaled form, one token tile and two
def test_w8_gemm_results_and_residuals_at_any_element(tokens):
    """Only x and the codes have to begin on 16 bytes."""
    from lemoq import _cabi

    codes, scale = _w8(256, 256, tokens)
    x = torch.randn(tokens, 256, generator=torch.Generator().manual_seed(5)).half()
    resid = torch.randn(tokens, 256, generator=torch.Generator().manual_seed(6)).half()
    ref = ops.dense_w8_gemv(x, codes, scale, 128).half() + resid
    dev = [t.to(DEV) for t in (x, codes, scale)]
    for y_at, resid_at in ((1, 0), (0, 1), (4, 4), (0, 0)):
        y = torch.full((tokens * 256 + 8,), float("nan"), dtype=torch.float16, device=DEV)
        held = torch.zeros(tokens * 256 + 8, dtype=torch.float16, device=DEV)
        held[resid_at: resid_at + tokens * 256] = resid.flatten().to(DEV)
        _cabi.call("lemoq_w8_gemm", _cabi.ptr(dev[0]), tokens, _cabi.ptr(dev[1]), _cabi.ptr(dev[2]), 256, 256, 128, None, 1, 0, 0,
                   _cabi.ptr(held) + 2 * resid_at, _cabi.ptr(y) + 2 * y_at, None, _cabi.current_stream())
        assert rel_err(y[y_at: y_at + tokens * 256].view(tokens, 256), ref) < PER_KERNEL_REL_TOL
        assert bool(y[:y_at].isnan().all()) and bool(y[y_at + tokens * 256:].isnan().all())


@pytest.mark.parametrize("counts,exact", [((0, 1, 16, 17, 0), True), ((70, 0, 3), True), ((128, 129, 0, 257, 1), False)])
def test_w8_gemm_segments(counts, exact):
    n, k, rows = 258, 256, sum(counts)
    codes, scale = _w8(n, k, rows, experts=len(counts))
    x = torch.randn(rows + 3, k, generator=torch.Generator().manual_seed(rows)).half()
    seg = torch.tensor([sum(counts[:e]) for e in range(len(counts) + 1)], dtype=torch.int32)
    got = _gemm(x.to(DEV), codes.to(DEV), scale.to(DEV), seg=seg.to(DEV), exact=exact)
    ref = torch.cat([ops.dense_w8_gemv(x[seg[e]: seg[e + 1]], codes[e], scale[e], 128) for e in range(len(counts)) if counts[e]])
    assert rel_err(got[:rows], ref) < PER_KERNEL_REL_TOL
    assert bool(got[rows:].isnan().all())  # rows of no expert are left alone


# prompts shorter than a tile of 128 query rows, one row into the second tile and into the second block; hidden 256 .. 512, 8 and 128 experts
@pytest.mark.parametrize("tokens,spec", [(2, dict(hidden=256, heads=2, experts=8, top_k=2, ffn=128)), (129, dict(hidden=256, heads=2, experts=8, top_k=2, ffn=128)),
                                         (257, dict(hidden=512, heads=4, experts=128, top_k=16, ffn=256))])
def test_prompt_matches_oracle(tokens, spec):
    from benchmarks.cudagraph import StaticCacheDecodeSession

    spec = glue.OlmoeSpec(layers=2, head_dim=128, vocab=512, **spec)
    wf = glue.random_float_weights(spec, seed=tokens, dtype=torch.float16, std=0.05, norm_weight_jitter=0.1)
    # a dominant residual stream and a decisive router: no top-k choice hangs on the last bit of an fp16 sum
    wf.embed.mul_(20.0)
    for layer in wf.layers:
        layer.router.mul_(5.0)
    wq = glue.quantize_weights(wf)
    model = lemoq_model_from_oracle(wf)
    install_canonical(model, tokens, 4)
    prompt = torch.tensor([[(11 * i * i + 3) % spec.vocab for i in range(tokens)]])
    state = glue.new_state(spec, tokens + 4)
    first = glue.prefill(wq, state, prompt[0])
    session = StaticCacheDecodeSession(model, prompt.to(DEV), ctx=tokens, max_new_tokens=4, engine="ops")
    assert "_lemoq_prompt_plan" in session.cache.__dict__ and int(session.cache._lemoq_prompt_plan["flags"]) == 0
    for i, slot in enumerate(session.cache.layers):
        assert rel_err(slot.keys[:, :, :tokens], state.keys[i][:, :, :tokens]) < 2e-2
        assert rel_err(slot.values[:, :, :tokens], state.values[i][:, :, :tokens]) < 2e-2
        assert not slot.keys[:, :, tokens:].any()
    logits = session.prefill().logits
    assert tuple(logits.shape) == (1, tokens, spec.vocab)
    assert rel_err(logits[0, -1], first) < 2e-2
    assert session.seed_token_id == int(first.float().argmax())


# one sequence; more sequences than a tile of tokens takes exactly; more heads than SMs
@pytest.mark.parametrize("sequences", [1, 5, 67])
def test_lockstep_matches_the_step_by_parts(sequences):
    """The native lockstep step against the same step written with the per-operator kernels."""
    from benchmarks.cudagraph import StaticCacheDecodeSession
    from benchmarks.expert_parallel import ExpertParallelDecoder

    spec = glue.OlmoeSpec(layers=2, hidden=512, heads=4, head_dim=128, experts=16, top_k=4, ffn=256, vocab=512)
    wf = glue.random_float_weights(spec, seed=sequences, dtype=torch.float16, std=0.05, norm_weight_jitter=0.1)
    wf.embed.mul_(20.0)
    for layer in wf.layers:
        layer.router.mul_(5.0)
    model = lemoq_model_from_oracle(wf)
    ctx = 140
    install_canonical(model, ctx, 8)
    prompt = torch.tensor([[(7 * i * i + 1) % spec.vocab for i in range(ctx)]], device=DEV)
    session = StaticCacheDecodeSession(model, prompt, ctx=ctx, max_new_tokens=8, engine="ops")
    decoders = [ExpertParallelDecoder(model, session, sequences=sequences, world=1, rank=0, static_exchange=True) for _ in range(2)]
    assert decoders[0].native is not None
    decoders[1].native = None
    tokens = (torch.arange(sequences, device=DEV) * 37 + 5) % spec.vocab
    with torch.no_grad():
        for _ in range(3):
            got, ref = (d.step(tokens) for d in decoders)
            # over all rows: now and then a sequence has another, nearly equal expert in its last slot
            assert float((got.float() - ref.float()).norm() / ref.float().norm()) < 5e-3
            tokens = ref.float().argmax(dim=-1)
    for a, b in zip(decoders[0].kv, decoders[1].kv):
        assert float((a["kc"] != b["kc"]).float().mean()) < 1e-2 and rel_err(a["vs"], b["vs"]) < 1e-2
    assert decoders[0].error_flags() == 0


def test_replaced_weights_are_the_ones_a_prompt_uses():
    """The tensors of a model may be exchanged between two prompts of a session, and between a step and its capture."""
    from benchmarks.cudagraph import StaticCacheDecodeSession
    from benchmarks.expert_parallel import ExpertParallelDecoder

    spec = glue.OlmoeSpec(layers=2, hidden=256, heads=2, head_dim=128, experts=8, top_k=2, ffn=128, vocab=512)
    wf = glue.random_float_weights(spec, seed=3, dtype=torch.float16, std=0.05, norm_weight_jitter=0.1)
    model, tokens = lemoq_model_from_oracle(wf), 40
    install_canonical(model, tokens, 4)
    prompt = torch.tensor([[(11 * i * i + 3) % spec.vocab for i in range(tokens)]], device=DEV)
    session = StaticCacheDecodeSession(model, prompt, ctx=tokens, max_new_tokens=4, engine="ops")
    decoder = ExpertParallelDecoder(model, session, sequences=2, world=1, rank=0, static_exchange=True)
    first = session.prefill().logits.clone()
    step = lambda d: (setattr(d, "position", tokens), d.step(torch.tensor([1, 2], device=DEV)).clone())[1]  # noqa: E731
    stepped = step(decoder)
    lm, norm = model.lm_head, model.model.layers[1].input_layernorm
    kept = norm.weight, lm.scale
    norm.weight, lm.scale = torch.nn.Parameter(-norm.weight.detach()), lm.scale * 2
    other, other_step = session.prefill().logits.clone(), step(decoder)
    fresh = StaticCacheDecodeSession(model, prompt, ctx=tokens, max_new_tokens=4, engine="ops")
    assert torch.equal(other, fresh.prefill().logits) and rel_err(other, first) > 0.5 and rel_err(other_step, stepped) > 0.5
    decoder.capture()
    assert torch.equal(step(decoder), other_step)
    norm.weight, lm.scale = kept
    torch.empty(1 << 20, dtype=torch.uint8, device=DEV).fill_(255)  # would land on freed weights
    assert torch.equal(step(decoder), other_step)  # a captured graph goes on with the weights it was captured with
    assert torch.equal(session.prefill().logits, first)


# the experts' scales are finer or coarser than the rest of the model's; the sizes are such that every kernel would take them
@pytest.mark.parametrize("group", [64, 256])
def test_experts_of_another_group_size_match_oracle(group):
    """Not a model that one native description fits: prompt, decode and lockstep step follow the experts' own group size all the same."""
    from benchmarks.cudagraph import StaticCacheDecodeSession
    from benchmarks.expert_parallel import ExpertParallelDecoder
    from benchmarks.runner import install_replacements
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts

    spec = glue.OlmoeSpec(layers=2, hidden=512, heads=4, head_dim=128, experts=8, top_k=2, ffn=512, vocab=512)
    wf = glue.random_float_weights(spec, seed=group, dtype=torch.float16, std=0.05, norm_weight_jitter=0.1)
    wf.embed.mul_(20.0)
    for layer in wf.layers:
        layer.router.mul_(5.0)
    wq, model, packed, tokens = glue.quantize_weights(wf), lemoq_model_from_oracle(wf), {}, 33
    for i, (lq, lw) in enumerate(zip(wq.layers, wf.layers)):
        parts = (*ops.rtn_quantize_w8(lw.gate_up_w, group), *ops.rtn_quantize_w8(lw.down_w, group))
        lq.experts = ops.QuantExperts(*parts, group)
        packed[i] = QuantFusedExperts(*(t.to(DEV).contiguous() for t in parts), 8, group)
    install_replacements(model, attn="kernel", moe="grouped", quant_cfg={"bit_width": "w8a16", "dequant": "fused", "group_size": 128}, rmsnorm="fused",
                         ctx=tokens, max_new_tokens=4, prequantized=packed)
    prompt = torch.tensor([[(11 * i * i + 3) % spec.vocab for i in range(tokens)]])
    state = glue.new_state(spec, tokens + 4)
    first = glue.prefill(wq, state, prompt[0])
    session = StaticCacheDecodeSession(model, prompt.to(DEV), ctx=tokens, max_new_tokens=4)
    assert rel_err(session.prefill().logits[0, -1], first) < 2e-2 and session.seed_token_id == int(first.float().argmax())
    decoder = ExpertParallelDecoder(model, session, sequences=1, world=1, rank=0, static_exchange=group % 128 == 0)
    glue.build_int8_mirror(state)
    ref = glue.decode_step(wq, state, session.seed_token_id, tokens)
    assert rel_err(decoder.step(torch.tensor([session.seed_token_id], device=DEV))[0], ref) < 2e-2
    assert rel_err(session.decode_eager().reshape(-1), ref) < 2e-2


def test_a_flagged_prompt_raises():
    """The kernels clamp a token id or a position that is out of range and flag it: the call says so and seeds nothing."""
    from benchmarks.cudagraph import StaticCacheDecodeSession
    from lemoq.model import StaticCache

    spec = glue.OlmoeSpec(layers=1, hidden=256, heads=2, head_dim=128, experts=8, top_k=2, ffn=128, vocab=512)
    model = lemoq_model_from_oracle(glue.random_float_weights(spec, seed=4, dtype=torch.float16))
    install_canonical(model, 20, 4)
    prompt = torch.arange(20, device=DEV).unsqueeze(0)
    session = StaticCacheDecodeSession(model, prompt.clone(), ctx=20, max_new_tokens=4, engine="ops")
    first = session.prefill().logits.clone()
    for bad in (spec.vocab, -1):
        session.prompt_ids[0, 7] = bad
        with pytest.raises(RuntimeError, match="token id outside the vocabulary"):
            session.prefill()
        with pytest.raises(RuntimeError, match="prefill must run"):
            session.seed_token_id
    session.prompt_ids[0, 7] = 7
    assert torch.equal(session.prefill().logits, first)  # the word is clean again
    with torch.no_grad():
        cache, slots = StaticCache(model.config, 24), torch.arange(20, device=DEV)
        assert torch.equal(model(prompt, past_key_values=cache, cache_position=slots).logits, first)
        for ids, at, told in ((prompt + spec.vocab, slots, "token id"), (prompt, slots + 5, "position")):
            with pytest.raises(RuntimeError, match=told):
                model(ids, past_key_values=cache, cache_position=at)


def test_a_prompt_is_counted_and_hooks_fire():
    from benchmarks.cudagraph import StaticCacheDecodeSession
    from lemoq.quant.linear import dequant_activity, reset_dequant_counters

    spec = glue.OlmoeSpec(layers=2, hidden=256, heads=2, head_dim=128, experts=8, top_k=2, ffn=128, vocab=512)
    model = lemoq_model_from_oracle(glue.random_float_weights(spec, seed=6, dtype=torch.float16, std=0.05))
    install_canonical(model, 20, 4)
    session = StaticCacheDecodeSession(model, torch.arange(20, device=DEV).unsqueeze(0), ctx=20, max_new_tokens=4, engine="ops")

    def counted():
        reset_dequant_counters(model)
        del session.cache._lemoq_prompt_plan
        logits = session.prefill().logits.clone()
        return dequant_activity(model), logits

    native, logits = counted()
    assert "_lemoq_prompt_plan" in session.cache.__dict__ and native["separate_calls"] == 9 and native["fallbacks"] == {"multi_token": 9}
    session.cache._lemoq_prompt_plan = seen = []
    handle = model.model.layers[1].self_attn.o_proj.register_forward_hook(lambda module, args, out: seen.append(tuple(out.shape)))
    by_modules, same = counted()
    assert seen == [(1, 20, 256)] and "_lemoq_prompt_plan" not in session.cache.__dict__
    assert by_modules == native and rel_err(logits, same) < 2e-2
    handle.remove()
    session.prefill()
    assert len(seen) == 1 and "_lemoq_prompt_plan" in session.cache.__dict__


def test_a_prompt_whose_operations_matter_goes_through_the_modules():
    from torch.utils._python_dispatch import TorchDispatchMode

    from benchmarks.cudagraph import StaticCacheDecodeSession

    class Seen(TorchDispatchMode):
        count = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.count += func is torch.ops.aten.index_copy_.default
            return func(*args, **(kwargs or {}))

    spec = glue.OlmoeSpec(layers=2, hidden=256, heads=2, head_dim=128, experts=8, top_k=2, ffn=128, vocab=512)
    model = lemoq_model_from_oracle(glue.random_float_weights(spec, seed=8, dtype=torch.float16, std=0.05))
    install_canonical(model, 20, 4)
    session = StaticCacheDecodeSession(model, torch.arange(20, device=DEV).unsqueeze(0), ctx=20, max_new_tokens=4, engine="ops")
    native = session.prefill().logits.clone()
    for mode in (Seen(), torch.autocast("cuda", dtype=torch.float16)):
        del session.cache._lemoq_prompt_plan
        with mode:
            logits = session.prefill().logits.clone()
        assert "_lemoq_prompt_plan" not in session.cache.__dict__ and rel_err(logits, native) < 2e-2
        assert not isinstance(mode, Seen) or mode.count == 4  # k and v rows of both layers
        assert torch.equal(session.prefill().logits, native) and "_lemoq_prompt_plan" in session.cache.__dict__


def _routed_session(tokens, shape, change=lambda weights, prompt: None):
    from benchmarks.cudagraph import StaticCacheDecodeSession

    shape = {"hidden": 256, "experts": 72, "top_k": 5, **shape}
    spec = glue.OlmoeSpec(layers=1, heads=shape["hidden"] // 128, head_dim=128, ffn=128, vocab=512, **shape)
    wf = glue.random_float_weights(spec, seed=tokens, dtype=torch.float16, std=0.05, norm_weight_jitter=0.1)
    wf.embed.mul_(20.0)
    wf.layers[0].router.mul_(5.0 * (256 / shape["hidden"]) ** 0.5)  # logits of about 4 and at most 16 whatever the width
    prompt = torch.randint(0, spec.vocab - 1, (1, tokens), generator=torch.Generator().manual_seed(tokens))
    change(wf, prompt)
    model = lemoq_model_from_oracle(wf)
    install_canonical(model, tokens, 4)
    return StaticCacheDecodeSession(model, prompt.to(DEV), ctx=tokens, max_new_tokens=4, engine="ops"), wf


def _native_and_by_modules(session):
    """Logits of the native prompt, those of the same prompt through the modules (which a hook asks for), and what their router saw."""
    native, seen = session.prefill().logits[0], []
    assert session.cache.__dict__.pop("_lemoq_prompt_plan", None) is not None
    session.model.model.layers[0].mlp.register_forward_pre_hook(lambda module, args: seen.append(args[0].flatten(0, -2)))
    by_modules = session.prefill().logits[0]
    assert "_lemoq_prompt_plan" not in session.cache.__dict__
    return native, by_modules, seen[0]


def _row_errors(got, ref):
    got, ref = got.float(), ref.float()
    return (got - ref).norm(dim=-1) / ref.norm(dim=-1)


# Of a row, 2-norm.  Hidden states, activations, results and logits of both sides are fp16 values, some ten roundings of up to 2^-11 each; and the
# logits of an expert and of the largest one may come out a step of fp16 apart, up to 2^-10 of them each, by which the expert's weight changes as
# exp does.  With another token's experts a row is off by 0.15 and more.
def _row_tol(logits):
    return 1e-2 + 2 * 2 ** -10 * logits.abs().amax(dim=-1)


# either side of 16 tokens (the blocks that route), one, two, four, eight and sixteen tokens a block that copies, and more tokens than those blocks take
@pytest.mark.parametrize("tokens,shape", [(t, {}) for t in (15, 16, 17, 610, 1201, 2405, 4800, 9999, 16384, 16385, 16390)] +
                         # rows shorter than a warp's stride and of more than 2048 values, one and 32 experts a token, 128 of them
                         [(17, dict(hidden=2048, experts=8, top_k=1)), (33, dict(hidden=1024, experts=128, top_k=32)),
                          (20, dict(hidden=4096, experts=64, top_k=8)), (18, dict(hidden=4096, experts=128, top_k=8)), (5, dict(hidden=128, experts=40, top_k=3)),
                          # more heads and tiles of 128 queries than SMs: two tiles a block of the attention, the last one ragged
                          (650, dict(hidden=4096, experts=8, top_k=1))])
def test_rows_of_a_prompt_reach_their_experts(tokens, shape):
    """Row by row against the prompt through the modules, but for tokens whose last expert is not clear."""
    session, wf = _routed_session(tokens, shape)
    native, by_modules, h = _native_and_by_modules(session)
    logits = h.float() @ wf.layers[0].router.to(DEV).float().T
    kept = logits.topk(session.model.config.num_experts_per_tok + 1, dim=-1).values
    clear = kept[:, -2] - kept[:, -1] > 2 ** -8 * logits.abs().amax(dim=-1)  # a few steps of an fp16 logit, and the errors of what goes into it
    assert clear.float().mean() > 0.5 and float(_row_tol(logits).max()) < 0.05
    assert bool((_row_errors(native, by_modules) < _row_tol(logits))[clear].all())


@pytest.mark.parametrize("tokens", [17, 300])
@pytest.mark.parametrize("alike", [1, 8, 72])  # sets of experts that are alike: all of them, nine each, none
def test_of_equal_logits_the_lowest_expert_is_taken(tokens, alike):
    def change(wf, prompt):
        router = wf.layers[0].router
        router.copy_(router[torch.arange(router.shape[0]) % alike])
        if alike == 1:
            router.zero_()

    session, wf = _routed_session(tokens, {}, change)
    native, by_modules, h = _native_and_by_modules(session)
    logits = (h.float() @ wf.layers[0].router.to(DEV).float().T)[:, :alike]
    # the five choices are the lowest of the nine that have the largest logit, so that one has to be clear (72: the fifth)
    kept = logits.topk(6 if alike == 72 else min(2, alike), dim=-1).values
    clear = kept[:, -2] - kept[:, -1] > 2 ** -8 * logits.abs().amax(dim=-1) if alike > 1 else torch.ones(tokens, dtype=torch.bool, device=DEV)
    assert clear.float().mean() > 0.5 and float(_row_tol(logits).max()) < 0.05
    assert bool((_row_errors(native, by_modules) < _row_tol(logits))[clear].all())


def test_a_token_whose_router_logits_overflow_keeps_to_its_row():
    """Their softmax has no numbers: the token's own row has none either, and the tokens before it get what they get without it."""
    rows = []
    for last in (0, 511):
        def change(wf, prompt):  # only token 511 has a first value, and hardly another one; it goes to expert 3 with more than fp16 holds
            wf.embed[:, 0] = wf.embed[511] = wf.layers[0].o_w[0] = wf.layers[0].router[:, 0] = 0
            wf.embed[511, 0], wf.layers[0].router[3, 0], prompt[0, -1] = 20, 60000, last

        rows.append(_routed_session(77, {}, change)[0].prefill().logits[0])
    assert bool(rows[0].isfinite().all()) and torch.equal(rows[0][:-1], rows[1][:-1]) and bool(rows[1][-1].isnan().all())
