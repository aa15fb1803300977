"""Float32 attention of single tokens, whose CTAs share out a token's keys: beside float64 and the kernel for portions."""

import pytest
import torch

gpu = pytest.mark.gpu


def test_how_many_ctas_share_a_token():
    from lite_lang_b200 import ops
    ctas = [ops.attn_f32_ctas(n, 12, 2, 1000, 148) for n in (1, 6, 7, 18, 19, 37, 38, 64)]
    assert ctas == [8, 8, 4, 4, 2, 2, 1, 1]
    assert ops.attn_f32_ctas(4, 34, 2, 1000, 148) == 0                 # 17 heads a kv head
    assert ops.attn_f32_ctas(64, 64, 8, 32, 148) == 0 and ops.attn_f32_ctas(64, 64, 8, 33, 148) == 1


@gpu
@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
@pytest.mark.parametrize("nh,nkv,hd,page,window,ctxs", [
    (6, 1, 128, 16, None, [0, 15, 16, 127, 128, 2049]), (32, 2, 64, 7, None, [1, 300, 511]), (3, 3, 128, 48, 100, [99, 100, 1000]),
    (9, 1, 64, 16, 17, [5, 700])])
def test_single_tokens(ctas, nh, nkv, hd, page, window, ctxs):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(nh + hd + len(ctxs))
    ints = dict(dtype=torch.int32, device="cuda")
    n = len(ctxs) + 1                                                   # one entry of padding
    per = [(c + page) // page for c in ctxs]
    k, v = (torch.randn(sum(per), nkv, page, hd, generator=g, device="cuda") for _ in range(2))
    table, at = torch.full((len(ctxs), max(per)), -1, dtype=torch.int32), 0
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(1)).int()
    for i, m in enumerate(per):
        table[i, :m] = order[at:at + m]
        at += m
    q = torch.randn(n, nh * hd + 4, generator=g, device="cuda")[:, :nh * hd]
    cu, ctx = torch.arange(n + 1, **ints), torch.tensor(ctxs + [0], **ints)
    slot, status = torch.tensor(list(range(len(ctxs))) + [-1], **ints), torch.zeros(1, **ints)
    outs = []
    for way in (0, ctas):
        out = torch.full((n, nh * hd), 7.0, device="cuda")
        ops.attn_f32(out, q, k, v, table.cuda(), cu, ctx, slot, [1] * n, nh, nkv, hd, page, window, hd ** -0.5, status, ctas=way)
        assert bool((out[-1] == 0).all())
        outs.append(out[:-1].double())
    assert int(status.item()) == 0
    want = torch.empty_like(outs[0])
    for i, c in enumerate(ctxs):
        keys, vals = (t[table[i, :per[i]].long()].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, :c + 1].double()
                      .repeat_interleave(nh // nkv, 0) for t in (k, v))
        scores = (q[i].double().view(nh, 1, hd) @ keys.transpose(1, 2))[:, 0] * hd ** -0.5
        if window:
            scores[:, :max(0, c - window + 1)] = float("-inf")
        want[i] = (scores.softmax(-1)[:, None] @ vals).reshape(-1)
    was, err = (float((o - want).norm() / want.norm()) for o in outs)
    # the same terms and sums of float32 in another order: a few roundings of 2^-24 of scores and sums
    assert err <= max(1.1 * was, 2.0 ** -22), (err, was)


@gpu
@pytest.mark.parametrize("ctas", [1, 4])
def test_single_tokens_of_numbers_that_are_not_finite(ctas):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    nh, nkv, hd, page, n = 4, 1, 64, 16, 300
    ints = dict(dtype=torch.int32, device="cuda")
    pages = (n + page - 1) // page
    k, v = (torch.randn(pages, nkv, page, hd, generator=g, device="cuda") for _ in range(2))
    k[3, 0, 2, 5], v[7, 0, 0, 9], v[12, 0, 3, 1] = float("inf"), float("inf"), float("nan")
    q = torch.randn(3, nh * hd, generator=g, device="cuda")
    table, ctx, slot = torch.arange(pages, **ints)[None], torch.tensor([40, 119, n - 1], **ints), torch.zeros(3, **ints)
    cu, status, outs = torch.arange(4, **ints), torch.zeros(1, **ints), []
    for way in (0, ctas):
        out = torch.empty(3, nh * hd, device="cuda")
        ops.attn_f32(out, q, k, v, table, cu, ctx, slot, [1] * 3, nh, nkv, hd, page, None, hd ** -0.5, status, ctas=way)
        outs.append(out)
    assert int(status.item()) == 0
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(outs[0]), kind(outs[1]))
    fin = torch.isfinite(outs[0])
    assert bool(fin.any()) and bool((~fin).any()) and float((outs[0] - outs[1])[fin].abs().max()) <= 1e-5
    table[0, 1] = pages + 5                                              # a page that does not exist is reported and left out
    ops.attn_f32(outs[0], q, k, v, table, cu, ctx, slot, [1] * 3, nh, nkv, hd, page, None, hd ** -0.5, status, ctas=ctas)
    assert int(status.item()) != 0
