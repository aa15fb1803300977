"""Which of its ways a portion of routed experts takes: rows off the 16-byte boundaries and the switch for library products included."""

import pytest
import torch

from test_nevurax import dev

gpu = pytest.mark.gpu


def _part(gated, gen):
    from lite_lang_b200.config import PartSpec
    from lite_lang_b200.parts import build_part
    p = dict(hidden_size=64, experts=6, top=2, expert_ff=48, shared_ff=24)
    if gated:
        p.update(gated=True, limit=7.0, swish_alpha=1.702)
    part = build_part("feed_forward", PartSpec("routed_experts", p, "mlp."))
    t = {name: (0.3 * torch.randn(*d.shape, generator=gen)).to(torch.bfloat16) for name, d in part.tensors().items()}
    t["router"] = (2.0 * torch.randn(6, 64, generator=gen)).to(torch.bfloat16)
    part.load(lambda rel: t.get(rel), torch.bfloat16, dev())
    return part


def _count(monkeypatch, ops, name):
    calls, real = [], getattr(ops, name)
    monkeypatch.setattr(ops, name, lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    return calls


@gpu
@pytest.mark.parametrize("gated", [False, True])
def test_ways(gated, monkeypatch):
    from lite_lang_b200 import ops
    from lite_lang_b200.parts import whole_output
    gen = torch.Generator().manual_seed(4)
    part = _part(gated, gen)
    x = torch.randn(150, 64, generator=gen).to(torch.bfloat16).to(dev())
    own, library = _count(monkeypatch, ops, "expert_products"), _count(monkeypatch, ops, "grouped_product")
    want = whole_output(part.forward(x, None), x.dtype)
    assert len(own) == 2 and not library
    # rows that start off the boundary, and rows of another stride: the same products, the same bits
    off = torch.empty(150 * 64 + 1, dtype=x.dtype, device=dev())[1:].view(150, 64).copy_(x)
    wide = torch.empty(150, 67, dtype=x.dtype, device=dev())[:, :64].copy_(x)
    for other in (off, wide):
        own.clear()
        assert torch.equal(whole_output(part.forward(other, None), x.dtype), want)
        assert len(own) == 2 and not library
    # library products
    monkeypatch.setattr(ops, "TC_ENABLED", False)
    own.clear()
    got = whole_output(part.forward(x, None), x.dtype)
    assert not own and len(library) == 2
    assert float((got.double() - want.double()).norm() / want.double().norm()) <= 1e-2
