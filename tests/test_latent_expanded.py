"""Latent attention of prompt portions with expanded keys and values, beside the same part in the latent space."""

import pytest
import torch

gpu = pytest.mark.gpu


def _part(params, seed):
    from lite_lang_b200 import ops
    from lite_lang_b200.config.spec import PartSpec
    from lite_lang_b200.parts.base import build_part
    import lite_lang_b200.parts  # noqa: F401
    ops.configure_matmul_precision()
    part = build_part("mixer", PartSpec("latent_attention", params))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    std = {"norm": 0.05, "bias": 0.5}

    def fetch(name):
        d = part.tensors()[name]
        t = torch.randn(d.shape, generator=g, device="cuda") * std.get(d.role, 0.06 if d.role == "matrix" else 0.06)
        return (t + 1.0 if d.role == "norm" else t).to(torch.bfloat16)

    part.load(fetch, torch.bfloat16, torch.device("cuda", 0))
    part.prepare(torch.device("cuda", 0), torch.bfloat16)
    return part


def _run(part, steps, page, seed, seen=None):
    """Outputs of the steps (lists of new tokens a request, 0: the request is not in the step) through one cache.  ``seen``:
    gets each step's input and the requests of its rows."""
    from lite_lang_b200.cache.manager import CacheManager, PagedGroupSpec
    from lite_lang_b200.cache.storage import CacheStorage
    from lite_lang_b200.engine.batch import BatchBuilder, StepEntry
    device, need = torch.device("cuda", 0), part.cache_need()
    total = [sum(s[i] for s in steps) for i in range(len(steps[0]))]
    manager = CacheManager([PagedGroupSpec(1, need.head_dim, need.window, 1, 0)],
                           [sum((n + page - 1) // page for n in total) + 4], page, len(total), max(total))
    storage = CacheStorage(manager, torch.bfloat16, device)
    storage.k[0].fill_(float("nan"))
    status = torch.zeros(1, dtype=torch.int32, device=device)
    builder = BatchBuilder(manager, max(sum(s) for s in steps), len(total), device, status)
    slots = [manager.open() for _ in total]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    outs = []
    for s in steps:
        entries = [StepEntry(slots[i], [0] * n) for i, n in enumerate(s) if n]
        for e in entries:
            assert manager.reserve(e.slot, manager.length(e.slot) + len(e.tokens))
        storage.sync()
        batch = builder.build(entries)
        x = torch.randn(batch.num_tokens, part.hidden_size, generator=g, device="cuda").to(torch.bfloat16)
        outs.append(part.forward(x, batch, storage.paged_view(0, 0, batch.slot_maps[0], True)))
        if seen is not None:
            seen.append((x, torch.tensor([slots.index(e.slot) for e in batch.entries for _ in e.tokens], device="cuda")))
        for e in entries:
            manager.advance(e.slot, manager.length(e.slot) + len(e.tokens))
        torch.cuda.synchronize()
    assert int(status.item()) == 0
    return [o.float().sum(0) if o.dim() == 3 else o.float() for o in outs]


# portions at the edges of 64-row pages and 128-row tiles, going on behind cached tokens, beside single tokens
_STEPS = [[[64, 129, 16], [1, 200, 70]], [[300, 17], [63, 1], [130, 90]]]


@gpu
@pytest.mark.parametrize("steps", _STEPS)
@pytest.mark.parametrize("page", [16, 4])
@pytest.mark.parametrize("params", [
    dict(hidden_size=256, heads=3, dim=96, rot_dim=32, vdim=128, kv_rank=64, window=100, rot_dims=32, eps=1e-6),
    dict(hidden_size=256, heads=2, dim=64, rot_dim=0, vdim=64, kv_rank=128, q_rank=64, sink=True, eps=1e-6),
    dict(hidden_size=192, heads=5, dim=48, rot_dim=16, vdim=64, kv_rank=96, rot_dims=8, rot_layout="half_split",
         channel_gate=True, eps=1e-6)])
def test_expanded_portions_equal_the_latent_space(params, page, steps, monkeypatch):
    from lite_lang_b200 import ops
    calls = []
    real = ops.attn_prefill_tc_rows
    monkeypatch.setattr(ops, "attn_prefill_tc_rows", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    part = _part(params, 5)
    got = _run(part, steps, page, 9)
    assert calls
    monkeypatch.setattr(type(part), "EXPAND_MIN_TOKENS", 1 << 30)
    calls.clear()
    want = _run(part, steps, page, 9)
    assert not calls
    for a, b in zip(got, want):
        # both round their operands to bfloat16 (8 bits) in different places: a few roundings of the row's largest number
        assert float((a - b).abs().max()) <= 1.6e-2 * float(b.abs().max())
        assert float((a - b).norm()) <= 1e-2 * float(b.norm())


def _exact(part, x):
    """The part's output for one request's tokens, float64, from the same stored weights."""
    H, d, r, R, n = part.H, part.d, part.r, part.R, x.shape[0]

    def f(t):
        return t.double()

    proj = f(x) @ f(part.w_in).t()
    q = proj[:, :H * (d + r)]
    if part.q_rank is not None:
        c = proj[:, :part.q_rank]
        q = (c / (c.pow(2).mean(1, keepdim=True) + part.eps).sqrt() * f(part.q_norm_w)) @ f(part.w_uq).t()
    q = q.reshape(n, H, d + r)
    c, kr = proj[:, part.kv_off:part.kv_off + R], proj[:, part.kv_off + R:part.kv_off + R + r]
    c = c / (c.pow(2).mean(1, keepdim=True) + part.eps).sqrt() * f(part.norm_w)
    half = part.rot_dims // 2
    angle = torch.arange(n, device=x.device, dtype=torch.float64)[:, None] * f(part.freq)[None, :half]
    cs, sn = angle.cos() * part.amplitude, angle.sin() * part.amplitude

    def turned(t):                       # [n, ..., r]
        t = t.clone()
        u = slice(0, half) if part.half_split else slice(0, 2 * half, 2)
        v = slice(half, 2 * half) if part.half_split else slice(1, 2 * half, 2)
        shape = (n,) + (1,) * (t.dim() - 2) + (half,)
        a, b, co, si = t[..., u].clone(), t[..., v].clone(), cs.view(shape), sn.view(shape)
        t[..., u], t[..., v] = a * co - b * si, b * co + a * si
        return t

    k = torch.cat([torch.einsum("nr,hdr->nhd", c, f(part.w_uk)), turned(kr)[:, None, :].expand(n, H, r)], dim=2)
    q = torch.cat([q[..., :d], turned(q[..., d:])], dim=2)
    s = torch.einsum("ihd,jhd->hij", q, k) * part.scale
    i, j = torch.arange(n, device=x.device)[:, None], torch.arange(n, device=x.device)[None, :]
    seen = (j <= i) & ((i - j < part.window) if part.window else True)
    s = s.masked_fill(~seen, float("-inf"))
    if part.sink:
        s = torch.cat([s, f(part.sink_w)[:, None, None].expand(H, n, 1)], dim=2)
    p = torch.softmax(s, dim=2)[:, :, :n]
    o = torch.einsum("hij,jhe->ihe", p, torch.einsum("nr,hre->nhe", c, f(part.w_uv_t))).reshape(n, -1)
    if part.channel_gate:
        o = o * torch.sigmoid(proj[:, part.gate_off:part.gate_off + o.shape[1]])
    return o @ f(part.w_o).t()


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


# 64 expanded rows (one page): their product with the expanded weights is this package's own (tcgen05 from 8,192 weight rows
# on, streaming where the inner size is a multiple of 256), which lets the attention start before the rows' table is made
@gpu
@pytest.mark.parametrize("params", [
    dict(hidden_size=256, heads=32, dim=64, rot_dim=64, vdim=128, kv_rank=512, rot_dims=64, eps=1e-6),
    dict(hidden_size=256, heads=2, dim=128, rot_dim=0, vdim=128, kv_rank=256, sink=True, eps=1e-6)])
@pytest.mark.parametrize("tokens", [64, 37])
def test_expanded_portions_behind_the_packages_own_products(params, tokens, monkeypatch):
    """Several layers queued behind a busy device, so that every kernel starts as early as it may."""
    from lite_lang_b200 import ops
    from lite_lang_b200.cache.manager import CacheManager, PagedGroupSpec
    from lite_lang_b200.cache.storage import CacheStorage
    from lite_lang_b200.engine.batch import BatchBuilder, StepEntry
    device, layers, calls = torch.device("cuda", 0), 6, []
    for name in ("gemm_tc", "gemm_stream"):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *a, _real=real, **k: (calls.append(tuple(a[1].shape)), _real(*a, **k))[1])
    parts = [_part(params, 20 + i) for i in range(layers)]
    need = parts[0].cache_need()
    manager = CacheManager([PagedGroupSpec(1, need.head_dim, need.window, layers, 0)], [8], 16, 1, tokens)
    storage = CacheStorage(manager, torch.bfloat16, device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    builder = BatchBuilder(manager, tokens, 1, device, status)
    slot = manager.open()
    assert manager.reserve(slot, tokens)
    storage.sync()
    batch = builder.build([StepEntry(slot, [0] * tokens)])
    x = torch.randn(tokens, 256, device=device, generator=torch.Generator(device="cuda").manual_seed(3)).to(torch.bfloat16)
    busy = torch.randn(8192, 8192, device=device, dtype=torch.bfloat16)

    def run():
        torch.cuda.synchronize()
        for _ in range(8):
            torch.mm(busy, busy)                                     # milliseconds: the launches below pile up behind it
        return [p.forward(x, batch, storage.paged_view(0, i, batch.slot_maps[0], True)) for i, p in enumerate(parts)]

    outs = run()
    assert sum(shape == tuple(p.w_kv.shape) for p in parts for shape in calls) >= layers, calls
    again = run()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for p, a, b in zip(parts, outs, again):
        assert torch.equal(a, b)
        # bfloat16 at each of five products and twice in the attention: a few 2^-9 of the result
        assert _rel(a.float().sum(0) if a.dim() == 3 else a, _exact(p, x)) <= 1.2e-2


# the last block of queries of these portions is short enough for the products that stream their weights, which here are
# rows that a kernel of the same step gathers: those must not be asked for before that kernel has written them
@gpu
@pytest.mark.parametrize("params", [
    dict(hidden_size=256, heads=2, dim=96, rot_dim=128, vdim=64, kv_rank=384, rot_dims=128, eps=1e-6),
    dict(hidden_size=256, heads=3, dim=64, rot_dim=0, vdim=128, kv_rank=256, window=100, eps=1e-6)])
@pytest.mark.parametrize("tokens", [258, 276])
def test_gathered_rows_are_not_streamed_as_weights(params, tokens, monkeypatch):
    from lite_lang_b200 import ops
    streamed, scored = [], []
    for name in ("gemm_tc", "gemm_stream"):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *a, _real=real, **k: (streamed.append(a[1].data_ptr()), _real(*a, **k))[1])
    gather = ops.latent_gather
    monkeypatch.setattr(ops, "latent_gather", lambda dst, *a, **k: (scored.append(dst.data_ptr()), gather(dst, *a, **k))[1])
    part = _part(params, 5)
    monkeypatch.setattr(type(part), "EXPAND_MIN_TOKENS", 1 << 30)
    got = _run(part, [[tokens]], 16, 9)[0]
    assert len(scored) == 2 and not set(scored) & set(streamed)
    x = torch.randn(tokens, part.hidden_size, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda")
    assert _rel(got, _exact(part, x.to(torch.bfloat16))) <= 1.2e-2


# single tokens, portions too short to be expanded in front of, between and behind long ones; then portions that go on
_MIXED = [[[1, 8, 100, 20, 300, 5, 31, 32], [40, 1, 33, 64, 2, 90, 1, 1]], [[0, 17, 17, 64], [64, 1, 200, 16]], [[16, 31], [31, 2]]]


@gpu
@pytest.mark.parametrize("steps", _MIXED)
@pytest.mark.parametrize("params", [
    dict(hidden_size=256, heads=3, dim=96, rot_dim=32, vdim=128, kv_rank=64, window=100, rot_dims=32, eps=1e-6),
    dict(hidden_size=256, heads=2, dim=64, rot_dim=0, vdim=64, kv_rank=128, q_rank=64, sink=True, eps=1e-6),
    dict(hidden_size=192, heads=5, dim=48, rot_dim=16, vdim=64, kv_rank=96, rot_dims=8, rot_layout="half_split",
         channel_gate=True, eps=1e-6)])
def test_portions_of_all_lengths_beside_float64(params, steps, monkeypatch):
    """No further off than the same portions in the latent space, with the long ones expanded, all at once or an entry at a
    time; those below 32 tokens never are."""
    from lite_lang_b200 import ops
    lens, real = [], ops.latent_unpage
    monkeypatch.setattr(ops, "latent_unpage", lambda *a, **k: (lens.append([n for _, n in a[5]]), real(*a, **k))[1])
    part, err = _part(params, 5), {}
    for way in ("latent", "expanded", "one by one"):
        monkeypatch.setattr(type(part), "EXPAND_MIN_TOKENS", 1 << 30 if way == "latent" else part.PRODUCT_MIN_TOKENS)
        if way == "one by one":
            monkeypatch.setattr(type(part), "EXPAND_BYTES", 1)
        lens.clear()
        seen = []
        outs = _run(part, steps, 16, 9, seen)
        long = sorted(n for s in steps for n in s if n >= 32)
        assert sorted(n for span in lens for n in span) == ([] if way == "latent" else long)
        assert way != "one by one" or all(len(span) == 1 for span in lens)
        got, want = [], []
        for i in range(len(steps[0])):
            x = torch.cat([x[who == i] for x, who in seen])
            got.append(torch.cat([o[who == i] for o, (_, who) in zip(outs, seen)]))
            want.append(_exact(part, x))
            # bfloat16 at each of five products and twice in the attention: a few 2^-9 of the result
            assert _rel(got[-1], want[-1]) <= 1.2e-2
        err[way] = _rel(torch.cat(got), torch.cat(want))
    assert max(err["expanded"], err["one by one"]) <= 1.15 * err["latent"], err
