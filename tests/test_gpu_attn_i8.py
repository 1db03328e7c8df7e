"""The tensor-core decode attention over the int8 mirror at the edges of its tiles of 128 positions, its splits and its persistent grid."""

from __future__ import annotations

import pytest
import torch

from gpu_util import PER_KERNEL_REL_TOL, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


# nothing filled; one position; either side of a tile; a last tile of one position in a split of its own; more heads than two blocks per SM
@pytest.mark.parametrize("heads,capacity,filled,splits", [(3, 40, 0, 1), (3, 40, 0, 4), (2, 40, 1, 3), (2, 200, 127, 2), (2, 200, 128, 2), (2, 200, 129, 2),
                                                          (5, 700, 641, 19), (5, 700, 700, 6), (300, 300, 259, 4), (700, 131, 131, 1),
                                                          # as many splits as are merged in one trip, one more, more than a warp has lanes
                                                          (2, 2600, 2560, 20), (2, 2700, 2561, 21), (3, 4300, 4225, 40)])
def test_attn_i8_edges(heads, capacity, filled, splits):
    from lemoq import _cabi

    g = torch.Generator().manual_seed(heads + filled)
    q = torch.randn(heads, 128, generator=g).half()
    kc, vc = (torch.randint(-127, 128, (heads, capacity, 128), generator=g, dtype=torch.int8) for _ in range(2))
    ks, vs = ((torch.rand(heads, capacity, generator=g) * 0.02 + 0.001).half() for _ in range(2))
    ks[:, filled:] = float("nan")  # scales behind the filled length need not be numbers
    vs[:, filled:] = float("nan")
    q[0] = 0
    dev = [t.to(DEV) for t in (q, kc, ks, vc, vs)]
    out = torch.full((heads, 128), float("nan"), dtype=torch.float16, device=DEV)
    ws = torch.zeros(int(_cabi.lib().lemoq_attn_workspace_bytes(heads, 128, splits)), dtype=torch.uint8, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    length = torch.tensor([filled], dtype=torch.int32, device=DEV)
    runs = []
    for _ in range(2):  # the second launch finds the arrival counters as the first left them
        _cabi.call("lemoq_attn_decode_int8", *(_cabi.ptr(t) for t in dev), capacity * 128, _cabi.ptr(length), _cabi.ptr(out), heads, capacity, 128, splits,
                   128 ** -0.5, _cabi.ptr(ws), _cabi.ptr(flag), _cabi.current_stream())
        runs.append(out.clone())
    assert int(flag) == 0 and torch.equal(runs[0], runs[1])
    if filled == 0:
        assert not out.any()
        return
    k, v = (c[:, :filled].double() * s[:, :filled].double()[..., None] for c, s in ((kc, ks), (vc, vs)))
    weights = torch.softmax(torch.einsum("hd,hsd->hs", q.double(), k) * 128 ** -0.5, dim=-1)
    assert rel_err(out, torch.einsum("hs,hsd->hd", weights, v)) < PER_KERNEL_REL_TOL


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
def test_query_at_any_element(offset):
    """A contiguous query may start anywhere in its storage (a slice of a projection row): every start gives what an aligned copy gives."""
    from lemoq.kernels.attn_decode import attn_decode_forward_int8

    g = torch.Generator().manual_seed(offset)
    codes, scales = torch.randint(-127, 128, (1, 3, 300, 128), generator=g, dtype=torch.int8).to(DEV), (torch.rand(1, 3, 300, generator=g) * 0.02).half().to(DEV)
    row = torch.randn(offset + 3 * 128, generator=g).half().to(DEV)
    q = row[offset:].view(1, 3, 1, 128)
    length = torch.tensor([290], dtype=torch.int32, device=DEV)
    got, ref = (attn_decode_forward_int8(x, codes, scales, codes, scales, length) for x in (q, q.clone()))
    assert rel_err(got, ref) < PER_KERNEL_REL_TOL


@pytest.mark.parametrize("what", ["q", "ks", "vs"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("filled", [40, 300])
def test_values_that_are_not_numbers_are_not_hidden(what, value, filled):
    """Digits cannot express them: the head they are in must come out as not finite, as the arithmetic has it, and no other head."""
    from lemoq.kernels.attn_decode import attn_decode_forward_int8

    g = torch.Generator().manual_seed(filled)
    t = {"q": torch.randn(1, 3, 1, 128, generator=g).half(), "kc": torch.randint(1, 128, (1, 3, 320, 128), generator=g, dtype=torch.int8),
         "ks": (torch.rand(1, 3, 320, generator=g) * 0.02).half()}
    t["vc"], t["vs"] = t["kc"].flip(2), t["ks"].flip(2)
    call = lambda: attn_decode_forward_int8(*(t[n].to(DEV) for n in ("q", "kc", "ks", "vc", "vs")), torch.tensor([filled], dtype=torch.int32, device=DEV)).cpu()  # noqa: E731
    ref = call()
    assert bool(ref.isfinite().all())
    t[what].view(3, -1)[1, 7] = value
    if what == "ks":
        t["q"][0, 1] = t["q"][0, 1].abs()  # the score is then plus infinity, not minus: such a position is not simply left out
    got = call()
    assert not got[0, 1].isfinite().any()
    assert torch.equal(got[0, 0], ref[0, 0]) and torch.equal(got[0, 2], ref[0, 2])
