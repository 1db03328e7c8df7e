"""The native call path of the short operators: same results as the path it shortcuts, at the token counts where the kernel changes."""

from __future__ import annotations

import pytest
import torch
from torch import nn

from gpu_util import PER_KERNEL_REL_TOL, rel_err
from oracle import lemoq_oracle as ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one expert for all tokens and experts without any; the sort's own gather (up to 1024 pairs) and the separate one behind it; ids out of range
@pytest.mark.parametrize("tokens,top_k,experts", [(1, 2, 4), (2, 1, 3), (5, 3, 7), (17, 8, 16), (130, 8, 16)])
def test_experts_for_several_tokens(tokens, top_k, experts):
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts, grouped_moe_forward_quant, grouped_moe_forward_quant_tokens

    hidden, ffn = 256, 384
    g = torch.Generator().manual_seed(tokens)
    gu, dn = (ops.rtn_quantize_w8(torch.randn(experts, *s, generator=g) * 0.05, 128) for s in ((2 * ffn, hidden), (hidden, ffn)))
    q = ops.QuantExperts(*gu, *dn, 128)
    x = torch.randn(tokens, hidden, generator=g).half()
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)])
    ids[0] = ids[0, 0]
    weights = torch.rand(tokens, top_k, generator=g).half()
    ref = torch.stack([ops.grouped_moe_w8(x[t], q, ids[t], weights[t])[0] for t in range(tokens)])
    ids[0] = torch.where(ids[0] == experts - 1, experts + 5, ids[0])  # clamped back to the last expert
    own = QuantFusedExperts(*(t.to(DEV) for t in (*gu, *dn)), 8, 128)
    args = x.to(DEV), own, ids.to(DEV), weights.to(DEV)
    got = grouped_moe_forward_quant_tokens(*args) if tokens > 1 else grouped_moe_forward_quant(args[0][0], own, args[2][0], args[3][0])
    assert rel_err(got, ref) < PER_KERNEL_REL_TOL


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("mode", ["fused", "separate"])
@pytest.mark.parametrize("shape", [(256,), (1, 1, 256), (1, 3, 256), (70, 256)])
def test_quant_linear_native_and_fallback_agree(mode, shape, bias):
    from lemoq.quant.linear import QuantLinear, SchemeSpec

    torch.manual_seed(len(shape))
    dense = nn.Linear(256, 130, bias=bias, device=DEV, dtype=torch.float16)
    linear = QuantLinear(dense, SchemeSpec.from_flags("w8a16", 128, dequant=mode))
    x = torch.randn(*shape, device=DEV).half()
    with torch.no_grad():
        got = linear(x)
        ref = torch.nn.functional.linear(x, linear.dequantized_weight(dtype=torch.float16), linear.bias)
        strided = linear(torch.cat([x, x], dim=-1)[..., :256])  # not contiguous: the Python way
    assert got.shape == ref.shape and rel_err(got, ref) < PER_KERNEL_REL_TOL and rel_err(strided, ref) < PER_KERNEL_REL_TOL
    single = x.numel() == 256
    assert single or not bias or torch.equal(got, ref)  # the bias is added before the one rounding
    assert linear._counters["fused_calls"] == (2 if single and mode == "fused" else 0)
    assert linear._counters["separate_calls"] == (0 if single and mode == "fused" else 2)
    assert linear._counters["fallbacks"] == ({"multi_token": 2} if mode == "fused" and not single else {})


def test_calls_leave_their_flags_where_the_host_sees_them():
    """The short calls pass no error word: clamped ids and lengths are in the device's status word, and a wait that ran out raises at the next
    call (the host sets the bit here: no kernel is made to wait)."""
    from ctypes import c_int

    from lemoq import _cabi
    from lemoq.kernels.attn_decode import attn_decode_forward_int8
    from lemoq.kernels.moe_grouped_quant import QuantFusedExperts, grouped_moe_forward_quant, grouped_moe_forward_quant_tokens
    from lemoq.quant.linear import QuantLinear, SchemeSpec

    g = torch.Generator().manual_seed(1)
    own = QuantFusedExperts(*(t.to(DEV) for s in ((256, 128), (128, 128)) for t in ops.rtn_quantize_w8(torch.randn(4, *s, generator=g), 128)), 8, 128)
    x, ids, weights = torch.randn(3, 128, generator=g).half().to(DEV), torch.tensor([[0], [3], [1]], device=DEV), torch.ones(3, 1, device=DEV).half()
    q, codes, scale = torch.randn(1, 2, 1, 128, device=DEV).half(), torch.ones(1, 2, 40, 128, dtype=torch.int8, device=DEV), torch.ones(1, 2, 40, device=DEV).half()
    linear = QuantLinear(nn.Linear(128, 64, bias=False, device=DEV, dtype=torch.float16), SchemeSpec.from_flags("w8a16", 128, dequant="fused"))
    calls = {"tokens": lambda n=0: grouped_moe_forward_quant_tokens(x, own, ids + n, weights), "token": lambda n=0: grouped_moe_forward_quant(x[0], own, ids[0] + n, weights[0]),
             "attention": lambda n=0: attn_decode_forward_int8(q, codes, scale, codes, scale, torch.tensor([40 + n], dtype=torch.int32, device=DEV)),
             "linear": lambda n=0: linear(x), "one": lambda n=0: linear(x[:1])}

    def flags():
        torch.cuda.synchronize()
        return _cabi.error_flags(clear=True)

    flags()
    with torch.no_grad():
        for name, call in calls.items():
            call()
            assert flags() == 0, name
            call(9)  # clamped, as ever
            assert flags() == {"tokens": _cabi.FLAG_BAD_EXPERT, "token": _cabi.FLAG_BAD_EXPERT, "attention": _cabi.FLAG_BAD_LENGTH}.get(name, 0), name
            c_int.from_address(_cabi.lib().lemoq_status_word()).value = _cabi.FLAG_WAIT_TIMEOUT | _cabi.FLAG_BAD_EXPERT
            with pytest.raises(RuntimeError, match="wait ran out"):
                call()
            call()
            assert flags() == _cabi.FLAG_BAD_EXPERT, name


class _Marked(torch.Tensor):
    """A tensor class whose operations have to be seen to keep it."""


def _jvp(f, x):
    import torch.autograd.forward_ad as fw

    with fw.dual_level():
        return fw.unpack_dual(f(fw.make_dual(x, x + 1))).tangent


def _autocast(f, x):
    with torch.autocast("cuda", dtype=torch.bfloat16):
        return f(x)


def _scale_gradient(f, x):
    with torch.enable_grad():
        scale = f.scale.detach().requires_grad_()
        f.scale = scale
        return torch.autograd.grad(f(x).float().square().mean(), scale)[0]


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("tokens", [4, 70])  # (vmap: two halves)
@pytest.mark.parametrize("way", [_jvp, _autocast, _scale_gradient, lambda f, x: torch.func.vmap(f)(x.view(2, -1, 256)).flatten(0, 1),
                                 lambda f, x: torch.func.jvp(f, (x,), (x + 1,))[1], lambda f, x: torch.jit.trace(f, (x + 1,), check_trace=False)(x),
                                 lambda f, x: f(x.as_subclass(_Marked)), lambda f, x: f(torch.cat([x.flatten()[:1], x.flatten()])[1:].view_as(x)),
                                 lambda f, x: torch.compile(f, backend="eager", fullgraph=True)(x)],
                         ids=["tangent", "autocast", "scale gradient", "vmap", "jvp", "trace", "subclass", "misaligned", "compile"])
def test_quant_linear_where_the_operation_itself_matters(way, tokens, bias):
    """What torch does with a linear it does with this one: the same result and kind of result as with the rebuilt weight."""
    from lemoq.quant.linear import QuantLinear, SchemeSpec

    class Rebuilt(QuantLinear):
        def forward(self, x):
            return torch.nn.functional.linear(x, self.dequantized_weight(dtype=x.dtype), self.bias)

    torch.manual_seed(tokens)
    dense = nn.Linear(256, 130, bias=bias, device=DEV, dtype=torch.float16)
    x = torch.randn(tokens, 256, device=DEV).half()
    with torch.no_grad():
        got, ref = (way(kind(dense, SchemeSpec.from_flags("w8a16", 128, dequant="fused")), x) for kind in (QuantLinear, Rebuilt))
    assert type(got) is type(ref) and got.dtype == ref.dtype and got.shape == ref.shape
    assert rel_err(got, ref) < (PER_KERNEL_REL_TOL if ref.dtype != torch.bfloat16 else 8 * PER_KERNEL_REL_TOL)


@pytest.mark.parametrize("int8", [True, False])
@pytest.mark.parametrize("before,heads", [("warm", 5), ("call", 6), ("nothing", 7)])
def test_attention_is_captured_after_a_call_of_its_shape(before, heads, int8):
    """``warm()`` or an ordinary call leaves the workspace that a capture needs; without either a capture is refused."""
    from lemoq.kernels.attn_decode import attn_decode_forward, attn_decode_forward_int8, warm
    from lemoq.kernels.kv_int8 import kv_int8_bulk_quantize

    heads += 20 * int8  # a shape of its own for every case
    g = torch.Generator(DEV).manual_seed(heads)
    q, k, v = (torch.randn(1, heads, n, 128, device=DEV, generator=g).half() for n in (1, 96, 96))
    filled = torch.tensor([70], dtype=torch.int32, device=DEV)
    cache = kv_int8_bulk_quantize(k, v)
    call = (lambda: attn_decode_forward_int8(q, cache["kc"], cache["ks"], cache["vc"], cache["vs"], filled)) if int8 else lambda: attn_decode_forward(q, k, v, filled)
    if before == "warm":
        warm(heads=heads, head_dim=128, kv_len=96)
    elif before == "call":
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    if before == "nothing":
        with pytest.raises(RuntimeError, match="before capture"), torch.cuda.graph(graph):
            call()
        return
    with torch.cuda.graph(graph):
        out = call()
    for _ in range(2):
        graph.replay()
        assert torch.equal(out, call())
        q.neg_()
