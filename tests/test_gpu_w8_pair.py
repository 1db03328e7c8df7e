"""The scaled W8 GEMM on pairs of SMs (more than 64 tokens, ``exact=False``) at the edges of its tiles, against the dequantised weights.

The tolerance is that of every fp16 operator: fp32 sums of fp16 products, one rounding of the weight (2^-11 of it) and one of the result."""

from __future__ import annotations

import pytest
import torch

from gpu_util import PER_KERNEL_REL_TOL, rel_err
from oracle import lemoq_oracle as ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weights(n, k, group, seed, experts=()):
    w = torch.randn(*experts, n, k, generator=torch.Generator().manual_seed(seed)) * 0.02
    codes, scale = ops.rtn_quantize_w8(w, group)
    return codes.to(DEV), scale.to(DEV), (codes.float().unflatten(-1, (-1, group)) * scale.float().unsqueeze(-1)).flatten(-2).to(DEV)


def _run(x, codes, scale, group, *, seg=None, gate_up=False, resid=None):
    from lemoq import _cabi

    n, k = codes.shape[-2:]
    y = torch.full((x.shape[0] + 1, n // 2 if gate_up else n), float("nan"), dtype=torch.float16, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    _cabi.call("lemoq_w8_gemm", _cabi.ptr(x), x.shape[0], _cabi.ptr(codes), _cabi.ptr(scale), n, k, group, _cabi.ptr(seg),
               codes.shape[0] if codes.dim() == 3 else 1, int(gate_up), 0, _cabi.ptr(resid), _cabi.ptr(y), _cabi.ptr(flag), _cabi.current_stream())
    assert int(flag) == 0 and bool(y[-1].isnan().all())
    return y[:-1]


def _swiglu(ref):
    gate, up = ref.chunk(2, dim=-1)
    return gate * torch.sigmoid(gate) * up


# tokens: either side of 64, 96, 128, 160 and 256 and of an odd number of 16-row boxes; rows: one, either side of 64, 128 and 256, off eight; groups of
# codes: one, odd, as many as the stages and more, rows of scales that do not fit the registers, scales over two groups of 128
@pytest.mark.parametrize("tokens", [65, 96, 97, 128, 129, 160, 161, 255, 257, 700])
@pytest.mark.parametrize("n,k,group", [(2, 128, 128), (66, 384, 128), (130, 640, 128), (258, 1024, 128), (2048, 2048, 128), (770, 1152, 128), (128, 2560, 256)])
def test_tiles(tokens, n, k, group):
    codes, scale, w = _weights(n, k, group, tokens + n)
    x = torch.randn(tokens, k, generator=torch.Generator().manual_seed(k)).half().to(DEV)
    resid = torch.randn(tokens, n, generator=torch.Generator().manual_seed(n)).half().to(DEV)
    ref = x.double() @ w.double().T
    assert rel_err(_run(x, codes, scale, group), ref) < PER_KERNEL_REL_TOL
    assert rel_err(_run(x, codes, scale, group, resid=resid), ref.half() + resid) < PER_KERNEL_REL_TOL
    assert rel_err(_run(x, codes, scale, group, gate_up=True), _swiglu(ref)) < 2 * PER_KERNEL_REL_TOL


@pytest.mark.parametrize("counts", [(0, 70, 1, 96, 33, 0), (160, 161, 0, 1, 159), (256, 257, 513, 0, 2), (40,) * 64, (0, 0, 300)])
def test_segments(counts):
    n, k = 258, 384
    codes, scale, w = _weights(n, k, 128, len(counts), (len(counts),))
    seg = torch.tensor([sum(counts[:e]) for e in range(len(counts) + 1)], dtype=torch.int32, device=DEV)
    x = torch.randn(sum(counts), k, generator=torch.Generator().manual_seed(7)).half().to(DEV)
    ref = torch.cat([x[seg[e]: seg[e + 1]].double() @ w[e].double().T for e in range(len(counts))])
    assert rel_err(_run(x, codes, scale, 128, seg=seg), ref) < PER_KERNEL_REL_TOL
    assert rel_err(_run(x, codes, scale, 128, seg=seg, gate_up=True), _swiglu(ref)) < 2 * PER_KERNEL_REL_TOL


# counts repeated: tiles of up to 160 tokens, some of more than 128 (all of the accumulator's columns) between some of fewer (a half in turn), and tiles
# of up to 96, all in halves; several tiles and more groups than stages a pair; rows: off 32, and gate/up rows off eight and off 32
@pytest.mark.parametrize("counts,k", [((20, 160, 130, 40, 97, 170), 640), ((20, 97, 60, 40), 896)])
@pytest.mark.parametrize("n", [264, 1008])
def test_accumulators_are_handed_over(counts, k, n):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    counts = counts * (1 + 2 * sms // (len(counts) * (n // 250)))  # four tiles a pair and more
    codes, scale, w = _weights(n, k, 128, n, (len(counts),))
    seg = torch.tensor(counts).cumsum(0).roll(1).tolist()
    seg = torch.tensor([0, *seg[1:], seg[0]], dtype=torch.int32, device=DEV)
    x = torch.randn(sum(counts), k, generator=torch.Generator().manual_seed(k)).half().to(DEV)
    resid = torch.randn(sum(counts), n, generator=torch.Generator().manual_seed(n)).half().to(DEV)
    refs = [part.double() @ w[e].double().T for e, part in enumerate(x.split(counts))]
    for kind, tol in (({}, 1), ({"resid": resid}, 1), ({"gate_up": True}, 2)):
        got = _run(x, codes, scale, 128, seg=seg, **kind).split(counts)
        for e, ref in enumerate(refs):  # each expert by itself: a wrong tile is not lost among right ones
            ref = _swiglu(ref) if "gate_up" in kind else ref.half() + resid[seg[e]: seg[e + 1]] if kind else ref
            assert rel_err(got[e], ref) < tol * PER_KERNEL_REL_TOL, (kind, e, counts[e])


def test_more_tiles_a_pair_than_are_looked_up_ahead():
    tokens = 256 * 66 * (torch.cuda.get_device_properties(0).multi_processor_count // 2) + 33
    codes, scale, w = _weights(2, 128, 128, 3)
    x = torch.randn(tokens, 128, device=DEV, generator=torch.Generator(DEV).manual_seed(3)).half()
    assert rel_err(_run(x, codes, scale, 128), x.float() @ w.T) < PER_KERNEL_REL_TOL
