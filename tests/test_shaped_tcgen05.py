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


def _exact(q, k, v, table, spans, nh, hd, mask, size, keep, sink, more, gates, page):
    """The portions' outputs in float64 (the first span is no portion)."""
    outs, at, nkv = [], spans[0][1], k.shape[1]
    for e, (c, n) in enumerate(spans[1:], 1):
        p, j = torch.arange(c, c + n, device="cuda")[:, None], torch.arange(c + n, device="cuda")[None, :]
        seen = j <= p
        if mask == "window":
            seen &= (p - j < size) | (j < keep)
        elif mask == "chunk":
            seen &= j // size == p // size
        pg = table[e][j[0] // page].long()
        keys, vals = (torch.where((pg < 0)[:, None, None], 0.0, t[pg.clamp(min=0), :, j[0] % page].double()) for t in (k, v))
        rows = torch.empty(n, nh, hd, dtype=torch.float64, device="cuda")
        for h in range(nh):
            s = q[at:at + n, h * hd:(h + 1) * hd].double() @ keys[:, h // (nh // nkv)].t() * hd ** -0.5
            if more["query_temperature"] is not None:
                coef, every = more["query_temperature"]
                s = s * (1 + coef * torch.log(((p + 1) // every + 1).double()))
            if more["softcap"]:
                s = more["softcap"] * torch.tanh(s / more["softcap"])
            if more["distance_bias"] is not None:
                s = s + more["distance_bias"].double()[(p - j).clamp(0, more["distance_bias"].shape[0] - 1), h]
            if more["distance_slope"] is not None:
                s = s - more["distance_slope"].double()[h] * (p - j)
            s = s.masked_fill(~seen, float("-inf"))
            if sink:
                extra = torch.zeros((), device="cuda") if more["sink_values"] is None else more["sink_values"][h]
                s = torch.cat([s, extra.double().expand(n, 1)], dim=1)
            rows[:, h] = torch.softmax(s, dim=1)[:, :c + n] @ vals[:, h // (nh // nkv)]
        if gates is not None:
            g = torch.sigmoid(gates[at:at + n].double())
            rows = rows * (g.view(n, nh, hd) if more["gate_channels"] else g[:, :, None])
        outs.append(rows.view(n, nh * hd) * more["out_scale"])
        at += n
    return torch.cat(outs)


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
    want = _exact(q, k, v, table, spans, nh, hd, mask, size, keep, sink, more, gates, page)
    was, err = (float((o.double() - want).norm() / want.norm()) for o in outs)
    # one rounding to bfloat16 (2^-9 at most, a third of that in the mean) on top of both, and sixteen-bit weights
    assert err <= max(1.1 * was, 2.0 ** -9), (err, was)
    # the same scores and sixteen-bit weights: what remains is the order of the sums and the one rounding to bfloat16
    assert float((outs[1] - outs[0]).abs().max()) <= 2.0 ** -7 * float(outs[0].abs().max())
    assert float((outs[1] - outs[0]).norm()) <= 2e-3 * float(outs[0].norm())


@pytest.mark.parametrize("params,spans,taken", [
    (dict(mask="window", mask_size=512, bias=True), [(0, 127)], False),
    (dict(mask="window", mask_size=512, bias=True), [(0, 128)], True),
    (dict(mask="window", mask_size=512, bias=True), [(0, 16), (120, 8), (0, 64)], True),
    (dict(mask="window", mask_size=20, bias=True), [(4000, 2000)], False),      # (a row block sees 19 keys and its own tokens)
    (dict(mask="window", mask_size=20, keep_first=100, bias=True), [(4000, 2000)], True),
    (dict(mask="causal", mask_size=None), [(0, 31), (0, 2)], False),
    (dict(mask="causal", mask_size=None), [(30, 2)], True),
    (dict(mask="chunk", mask_size=256), [(256, 20)], False),
    (dict(mask="chunk", mask_size=256), [(255, 20)], True)])
def test_which_shaped_portions_go_to_tcgen05(params, spans, taken):
    from lite_lang_b200.parts.modulated_attention import ModulatedAttention
    part = ModulatedAttention.__new__(ModulatedAttention)
    part.mask, part.mask_size, part.keep_first = params["mask"], params["mask_size"], params.get("keep_first", 0)
    part.bias_by_distance = torch.zeros(1) if params.get("bias") else None
    assert part._tc_preferred(spans, 7) is taken


# on both sides of the lines: which kernel a part's portion takes, and that a layer with other kv heads plans for itself
@gpu
@pytest.mark.parametrize("bias,tokens,taken", [(True, 127, False), (True, 128, True), (False, 31, False), (False, 32, True)])
def test_parts_take_the_kernel_that_is_meant(bias, tokens, taken, monkeypatch):
    from lite_lang_b200 import ops
    from lite_lang_b200.cache.manager import CacheManager, PagedGroupSpec
    from lite_lang_b200.cache.storage import CacheStorage
    from lite_lang_b200.config.spec import PartSpec
    from lite_lang_b200.engine.batch import BatchBuilder, StepEntry
    from lite_lang_b200.parts.base import build_part
    import lite_lang_b200.parts  # noqa: F401
    ops.configure_matmul_precision()
    device, names = torch.device("cuda", 0), []
    for name in ("attn_prefill_tc_shaped", "attn_shaped"):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *a, _real=real, _name=name, **k: (names.append(_name), _real(*a, **k))[1])
    g = torch.Generator(device="cuda").manual_seed(4)
    part = build_part("mixer", PartSpec("modulated_attention", dict(
        hidden_size=128, num_heads=4, num_kv_heads=2, head_dim=64, scale=0.125, mask="window", mask_size=200, sink="learned",
        distance_bias=dict(max=400.0, buckets=32) if bias else None)))
    part.load(lambda n: (torch.randn([32 if d is None else d for d in part.tensors()[n].shape], generator=g, device="cuda") * 0.1)
              .to(torch.bfloat16), torch.bfloat16, device)
    part.prepare(device, torch.bfloat16)
    manager = CacheManager([PagedGroupSpec(2, 64, 200, 1, 64)], [64], 16, 1, tokens)
    storage, status = CacheStorage(manager, torch.bfloat16, device), torch.zeros(1, dtype=torch.int32, device=device)
    slot = manager.open()
    assert manager.reserve(slot, tokens)
    storage.sync()
    x, outs = torch.randn(tokens, 128, generator=g, device="cuda").to(torch.bfloat16), []
    for least in (None, 1 << 30):                       # as meant, and by the other kernel
        if least:
            monkeypatch.setattr(type(part), "TC_MIN_KEYS", least)
            monkeypatch.setattr(type(part), "TC_MIN_KEYS_BIAS", least)
        batch = BatchBuilder(manager, tokens, 1, device, status).build([StepEntry(slot, [0] * tokens)])
        out = part.forward(x, batch, storage.paged_view(0, 0, batch.slot_maps[0], True))
        outs.append(out.float().sum(0) if out.dim() == 3 else out.float())
    assert names == ["attn_prefill_tc_shaped" if taken else "attn_shaped", "attn_shaped"]
    assert int(status.item()) == 0
    assert float((outs[0] - outs[1]).norm()) <= 1e-2 * float(outs[1].norm())
