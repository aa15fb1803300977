"""The grouped experts' small kernels at the sizes where they can go wrong: order of the pairs, activation of rows, sum."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,top,hidden,with_base", [(1, 1, 8, True), (33, 4, 264, False), (7, 9, 3592, True), (5, 5, 37, True)])
def test_combine(dtype, tokens, top, hidden, with_base):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(hidden)
    rows = tokens * top + 3
    y = torch.randn(rows, hidden, generator=g, device="cuda").to(dtype)
    base = torch.randn(tokens, hidden, generator=g, device="cuda").to(dtype) if with_base else None
    pair = torch.randint(-1, rows, (tokens, top), generator=g, device="cuda").to(torch.int32)
    got = ops.moe_combine(base, y, pair)
    want = torch.zeros(tokens, hidden, device="cuda")
    for k in range(top):                                # the same float32 sums in the same order
        want = want + torch.where(pair[:, k, None] >= 0, y[pair[:, k].clamp(min=0).long()].float(), 0.0)
    if with_base:
        want = want + base.float()
    assert torch.equal(got, want.to(dtype))


@gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,ff", [(1, 8), (5, 1032), (9, 2056), (130, 37)])
@pytest.mark.parametrize("limit,weights", [(0.0, True), (7.0, False)])
def test_row_gated_activation(dtype, rows, ff, limit, weights):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(rows + ff)
    h = (torch.randn(rows, 2 * ff, generator=g, device="cuda") * 4).to(dtype)
    w = torch.rand(rows, generator=g, device="cuda") if weights else None
    got = ops.moe_row_gated_act(h, w, limit, 1.702)
    a, b = h[:, :ff].double(), h[:, ff:].double()
    want = (a.clamp(max=limit) * torch.sigmoid(1.702 * a.clamp(max=limit)) * (b.clamp(-limit, limit) + 1) if limit
            else a * torch.sigmoid(a) * b)
    if weights:
        want = want * w.double()[:, None]
    # one rounding to the type (2^-9 of a bfloat16) after float32 arithmetic with an exponential (some 2^-20)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
    assert bool(((got.double() - want).abs() <= eps * want.abs() + 1e-6).all())


@gpu
@pytest.mark.parametrize("tokens,top,E", [(1, 1, 1), (300, 4, 16), (517, 3, 33), (2048, 2, 256), (40, 2, 32)])
def test_sort(tokens, top, E):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(E)
    idx = torch.randint(-1, E, (tokens, top), generator=g, device="cuda").to(torch.int32)
    w = torch.rand(tokens, top, generator=g, device="cuda")
    ends, row_token, row_w, pair_row = ops.moe_sort(idx, w, E)
    flat, pair = idx.reshape(-1).long(), pair_row.reshape(-1).long()
    on = flat >= 0
    counts = torch.bincount(flat[on], minlength=E) + 1
    assert torch.equal(ends.long(), torch.cumsum(counts, 0))
    assert bool((pair[~on] == -1).all()) and len(set(pair[on].tolist())) == int(on.sum())
    starts = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), ends.long()[:-1]])
    assert bool(((pair[on] > starts[flat[on]]) & (pair[on] < ends.long()[flat[on]])).all())
    assert torch.equal(row_token.long()[pair[on]], torch.arange(tokens * top, device="cuda")[on] // top)
    assert torch.equal(row_w[pair[on]], w.reshape(-1)[on])
    assert bool((row_w[starts] == 0).all()) and bool((row_token[starts] == 0).all())
    assert bool((row_w[int(ends[-1]):] == 0).all()) and bool((row_token[int(ends[-1]):] == 0).all())
