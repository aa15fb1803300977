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


def _run(part, steps, page, seed):
    """Outputs of the steps (lists of new tokens a request, 0: the request is not in the step) through one cache."""
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
