"""Experts' activation and routing weights in the epilogue of the streaming product: the same bits as the product and the activation
kernel after it, at the edges of units and of the token tiles, with experts that nobody chose holding what must not come through."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("act,weight_in", [("relu2", False), ("silu", False), ("gelu_tanh", True), ("gelu", False)])
@pytest.mark.parametrize("n,shared,ff,E,k", [(1, 0, 1024, 8, 128), (8, 96, 1350, 6, 384), (9, 520, 968, 8, 256), (17, 0, 4100, 2, 1536),
                                             (32, 8192, 0, 0, 128), (5, 7, 61, 3, 128)])
def test_same_bits_as_the_activation_kernel(n, shared, ff, E, k, act, weight_in):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(n * 100 + E)
    width = shared + E * ff
    x = torch.randn(n, k + 8, generator=g, device="cuda").to(torch.bfloat16)[:, :k]
    w = (torch.randn(width, k, generator=g, device="cuda") * k ** -0.5).to(torch.bfloat16)
    gates = torch.rand(n, E, generator=g, device="cuda")
    gates[torch.rand(n, E, generator=g, device="cuda") < 0.6] = 0.0
    if E > 1:
        gates[:, 1] = 0.0
        w[shared + ff] = float("inf")                       # of an expert that nobody chose
    got = ops.expert_hidden(x, w, gates, shared, ff, E, act, weight_in)
    want = ops.linear(x, w)
    ops.moe_act(want, gates, shared, ff, E, act, weight_in)
    assert torch.equal(got, want) and bool(torch.isfinite(got.float()).all())
