"""Shaped scores of prompt portions on the tcgen05 kernel, beside the mma.sync kernel that makes the same scores."""

import pytest
import torch

gpu = pytest.mark.gpu

_SHAPES = [
    dict(mask="causal", mask_size=None, sink=False, softcap=4.0, query_temperature=(0.3, 16)),
    dict(mask="window", mask_size=70, sink=True, keep_first=40, bias=200, learned=True, gate="channel"),
    dict(mask="window", mask_size=64, sink=True, keep_first=130, slope=True, gate="head"),
    dict(mask="chunk", mask_size=100, sink=True, slope=True, gate="channel"),
    dict(mask="causal", mask_size=None, sink=False, bias=33, out_scale=0.5),
    dict(mask="window", mask_size=7, sink=False, keep_first=3),
]


@gpu
@pytest.mark.parametrize("shape", _SHAPES)
@pytest.mark.parametrize("hd,nh,nkv", [(128, 14, 2), (64, 3, 3)])
@pytest.mark.parametrize("splits", [False, True])
def test_shaped_scores_equal_the_other_kernels(shape, hd, nh, nkv, splits):
    from lite_lang_b200 import ops
    shape, page = dict(shape), 16
    g = torch.Generator(device="cuda")
    g.manual_seed(hd + nh)
    spans = [(0, 1), (0, 65), (33, 200), (300, 18), (513, 127)]          # (cached, new); the first one is not a portion
    size, keep = shape["mask_size"], shape.pop("keep_first", 0)
    pages = [(c + n + page - 1) // page for c, n in spans]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(2)).tolist()
    k = torch.full((sum(pages) + 3, nkv, page, hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    v = k.clone()
    table = torch.full((len(spans), max(pages)), -1, dtype=torch.int32)
    for e, (c, n) in enumerate(spans):
        first = max(0, c - size + 1) if shape["mask"] == "window" else c // size * size if shape["mask"] == "chunk" else 0
        for lp in range(pages[e]):
            if (lp + 1) * page <= first and lp * page >= keep:
                continue                                                # given back
            table[e, lp] = pg = order.pop()
            live = min(page, c + n - lp * page)
            k[pg, :, :live] = torch.randn(nkv, live, hd, generator=g, device="cuda").to(torch.bfloat16)
            v[pg, :, :live] = torch.randn(nkv, live, hd, generator=g, device="cuda").to(torch.bfloat16)
    total = sum(n for _, n in spans)
    q = (torch.randn(total, nh * hd + 8, generator=g, device="cuda") * 2).to(torch.bfloat16)
    ints = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.cumsum(torch.tensor([n for _, n in spans]), 0).tolist(), **ints)[1:]
    ctx, slot, table = torch.tensor([c for c, _ in spans[1:]], **ints), torch.tensor([1, 2, 3, 4], **ints), table.to("cuda")
    rnd = dict(generator=g, device="cuda")
    bias, gate, learned = shape.pop("bias", 0), shape.pop("gate", None), shape.pop("learned", False)
    more = dict(keep_first=keep, sink_values=torch.randn(nh, **rnd) if learned else None,
                distance_bias=torch.randn(bias, nh, **rnd) if bias else None,
                distance_slope=torch.rand(nh, **rnd) * 0.1 if shape.pop("slope", False) else None,
                softcap=shape.pop("softcap", None), query_temperature=shape.pop("query_temperature", None),
                gate_channels=gate == "channel", out_scale=shape.pop("out_scale", 1.0))
    gates = None if gate is None else torch.randn(total, nh * hd if gate == "channel" else nh, **rnd).to(torch.bfloat16)
    status, outs, group = torch.zeros(1, **ints), [], nh // nkv
    rest = [(c, n) for c, n in spans[1:]]
    mask, sink = shape["mask"], shape["sink"]
    for way in (0, 1):
        out = torch.full((total, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        if way:
            plan = ops.attn_prefill_tc_plan(rest, group, size if mask == "window" else None, nkv,
                                            2 * ops.sm_count(q.device) if splits else 0, size if mask == "chunk" else None, keep)
            if splits:
                plan = (plan[0], 4, 2)
            ops.attn_prefill_tc_shaped(out, q, q.stride(0), gates, k, v, table, cu, ctx, slot, 4, plan, nh, nkv, hd, page, mask,
                                       size, sink, hd ** -0.5, status, **more)
        else:
            ops.attn_shaped(out, q, q.stride(0), False, gates, None, k, v, table, cu, ctx, slot, 4,
                            ops.attn_shaped_blocks([n for _, n in rest], group), nh, nkv, hd, hd, page, mask, size, sink,
                            hd ** -0.5, status, **more)
        assert int(status.item()) == 0
        assert bool((out[0] == 7.0).all())
        outs.append(out[1:].float())
    # the same scores and sixteen-bit weights: what remains is the order of the sums and the one rounding to bfloat16
    assert float((outs[1] - outs[0]).abs().max()) <= 2.0 ** -7 * float(outs[0].abs().max())
    assert float((outs[1] - outs[0]).norm()) <= 2e-3 * float(outs[0].norm())
