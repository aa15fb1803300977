"""The router of long portions on tensor cores beside float64: outputs at the edges of tiles, tokens at those of blocks, every score
form, an infinity in one token."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("E,top,shared,score", [(8, 2, False, "softmax"), (16, 4, True, "softmax_top"), (32, 3, False, "sigmoid"),
                                                (31, 5, True, "softmax"), (5, 5, False, "softmax"), (9, 2, False, "sigmoid"), (23, 4, True, "softmax")])
# (on tensor cores from 256 tokens on with 17 to 24 outputs, 297 with 11 to 16 or more than 24, 445 with 9 or 10, 4,096 with fewer)
@pytest.mark.parametrize("tokens,hidden", [(256, 16), (259, 528), (297, 528), (445, 16), (515, 528), (2048, 1536), (4099, 144)])
def test_logits_choice_and_weights(E, top, shared, score, tokens, hidden):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(E * 1000 + tokens + hidden)
    x = torch.randn(tokens, hidden + 8, generator=g, device="cuda").to(torch.bfloat16)[:, :hidden]
    w = torch.randn(E + shared, hidden, generator=g, device="cuda") * hidden ** -0.5
    bias = torch.randn(E, generator=g, device="cuda") * 0.1
    gates = torch.empty(tokens, E, device="cuda")
    idx, wts = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
    sw = torch.empty(tokens, device="cuda") if shared else None
    ops.moe_router(x, w, gates, idx, wts, top, score, bias=bias, shared_w=sw)
    z = x.double() @ w.double().T
    if shared:
        assert float((sw.double() - torch.sigmoid(z[:, E])).abs().max()) <= 1e-6
    z = z[:, :E] + bias.double()
    p = torch.softmax(z, -1) if score == "softmax" else torch.sigmoid(z) if score == "sigmoid" else z
    best = torch.topk(p, top, -1)
    clear = (torch.sort(p, -1, descending=True).values[:, :top + 1].diff(dim=-1).abs().min(-1).values > 1e-5) if top < E else \
        (torch.sort(p, -1, descending=True).values.diff(dim=-1).abs().min(-1).values > 1e-5)
    assert float(clear.double().mean()) > 0.9
    assert torch.equal(idx[clear].long(), best.indices[clear])
    want = torch.softmax(best.values, -1) if score == "softmax_top" else best.values
    # (float32 sums of `hidden` products and an exponential: a few units of the last place of numbers up to 1)
    assert float((wts[clear].double() - want[clear]).abs().max()) <= 3e-6
    dense = torch.zeros_like(p).scatter(1, best.indices, want)
    assert float((gates[clear].double() - dense[clear]).abs().max()) <= 3e-6


@gpu
@pytest.mark.parametrize("tokens", [300, 600])
def test_an_infinity_stays_in_its_token(tokens):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.randn(tokens, 64, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(16, 64, generator=g, device="cuda")
    x[37, 5] = float("inf")
    out = []
    for xs in (x, x[32:48].contiguous()):      # (the second: few tokens, the other kernel)
        n = xs.shape[0]
        gates = torch.empty(n, 16, device="cuda")
        idx, wts = torch.empty(n, 4, dtype=torch.int32, device="cuda"), torch.empty(n, 4, device="cuda")
        ops.moe_router(xs, w, gates, idx, wts, 4, "sigmoid")
        out.append((gates, idx, wts))
    assert torch.equal(out[0][1][32:48], out[1][1])
    assert torch.isfinite(out[0][0]).all() and float((out[0][2][32:48] - out[1][2]).abs().max()) <= 1e-6
