"""Experts of one or two tokens from the chosen experts' matrices only, beside float64."""

import pytest
import torch

gpu = pytest.mark.gpu


def test_which_steps_read_the_chosen_experts_only():
    from lite_lang_b200 import ops
    took = {(top, E): [[m for m in range(1, 9) if ops.experts_few_preferred(m, top, E, gated)] for gated in (False, True)] for top, E in ((4, 16), (2, 8), (8, 64), (1, 2), (6, 8))}
    assert took == {(4, 16): [[1], [1, 2]], (2, 8): [[1], [1, 2]], (8, 64): [[1], [1, 2]], (1, 2): [[1], [1]], (6, 8): [[], []]}
    assert not ops.experts_few_supported(*(torch.zeros(8, 8, dtype=torch.bfloat16) for _ in range(3)), 0, 8, 1)      # (not on a CUDA device)


@gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("M,K,N,shared,ff,E,top", [
    (1, 64, 40, 0, 8, 3, 1), (2, 1536, 1536, 64, 128, 16, 4), (1, 520, 33, 24, 72, 5, 2), (2, 3584, 257, 0, 56, 256, 8), (2, 2048, 100, 40, 264, 8, 8)])
def test_experts_of_few_tokens(M, K, N, shared, ff, E, top, gated):
    from lite_lang_b200 import ops
    M = M if gated else 1
    g = torch.Generator(device="cuda").manual_seed(M * K + E)
    rnd = dict(generator=g, device="cuda")
    width = shared + E * ff
    x = torch.randn(M, K + 8, **rnd).bfloat16()[:, :K]
    w_up = (torch.randn((2 if gated else 1) * width, K, **rnd) * K ** -0.5).bfloat16()
    w_down = (torch.randn(N, width, **rnd) * 0.1).bfloat16()
    gates = torch.zeros(M, E, device="cuda")
    for t in range(M):
        gates[t, torch.randperm(E, generator=torch.Generator().manual_seed(t))[:top].cuda()] = torch.rand(top, **rnd) + 0.1
    dead = (gates == 0).all(0).nonzero()[:, 0].tolist()
    for e in dead:                                                   # never read: would show
        a = (2 if gated else 1)
        w_up[a * (shared + e * ff):a * (shared + (e + 1) * ff)] = float("nan")
        w_down[:, shared + e * ff:shared + (e + 1) * ff] = float("nan")
    shared_w = torch.rand(M, **rnd) if gated and shared else None
    kind = dict(act=None, limit=3.0, shared_limit=2.0, alpha=1.702) if gated else dict(act="silu", weight_in=bool(shared))
    assert ops.experts_few_supported(x, w_up, w_down, shared, ff, E)
    out = ops.experts_few(x, w_up, w_down, gates, shared_w, shared, ff, E, **kind)
    assert out.shape == (1, M, N) and out.dtype == torch.float32
    want, xd = torch.zeros(M, N, dtype=torch.float64, device="cuda"), x.double()
    for e in ([-1] if shared else []) + [e for e in range(E) if e not in dead]:
        a, f = (shared + e * ff, ff) if e >= 0 else (0, shared)
        weight = gates[:, e].double() if e >= 0 else torch.ones(M, device="cuda").double() if shared_w is None else shared_w.double()
        if gated:
            lim = 3.0 if e >= 0 else 2.0
            y = (xd @ w_up[2 * a:2 * a + 2 * f].double().t()).bfloat16().double()
            left, right = y[:, :f].clamp(max=lim), y[:, f:].clamp(-lim, lim)
            h = left * torch.sigmoid(1.702 * left) * (right + 1) * weight[:, None]
        else:
            z = (xd @ w_up[a:a + f].double().t()).bfloat16().double()
            h = torch.nn.functional.silu(z * weight[:, None]) if shared else torch.nn.functional.silu(z) * weight[:, None]
        want += torch.where(weight[:, None] != 0, h, 0.0).bfloat16().double() @ w_down[:, a:a + f].double().t()
    # roundings of products and hidden units to bfloat16 on both sides, which may differ by one of 2^-8 where a float32 sum lies near
    # the middle: a small share of them
    assert float((out[0].double() - want).norm()) <= 2.0 ** -9 * float(want.norm())


@gpu
@pytest.mark.parametrize("M,K,gated", [(1, 24576, False), (1, 24440, True), (2, 12288, True), (2, 12208, True)])
def test_the_widest_rows(M, K, gated):
    """Rows that fill the shared memory of a block: the sizes that `experts_few_supported` ends at."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K)
    E, ff, N = 8, 16, 24
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w_up = (torch.randn((2 if gated else 1) * E * ff, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    w_down = torch.randn(N, E * ff, generator=g, device="cuda").bfloat16()
    gates = torch.zeros(M, E, device="cuda")
    gates[:, 2], gates[:, 5] = 0.75, 0.5
    assert ops.experts_few_supported(x, w_up, w_down, 0, ff, E)
    kind = dict(act=None, limit=7.0, alpha=1.702) if gated else dict(act="silu")
    out = ops.experts_few(x, w_up, w_down, gates, None, 0, ff, E, **kind)
    y = (x.double() @ w_up.double().t()).bfloat16().double().view(M, E, -1)
    if gated:
        left, right = y[..., :ff].clamp(max=7.0), y[..., ff:].clamp(-7.0, 7.0)
        h = left * torch.sigmoid(1.702 * left) * (right + 1)
    else:
        h = torch.nn.functional.silu(y)
    want = (h * gates.double()[..., None]).bfloat16().double().view(M, -1) @ w_down.double().t()
    assert float((out[0].double() - want).norm()) <= 2.0 ** -9 * float(want.norm())      # (as above)


@gpu
@pytest.mark.parametrize("K,N,shared,ff,E,top", [(1536, 1536, 1792, 1792, 16, 4), (512, 40, 0, 264, 16, 2), (256, 33, 40, 24, 64, 8)])
def test_a_token_beside_others(K, N, shared, ff, E, top):
    """One token's numbers are the same, whatever the other token of the step has chosen, and alone."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K + E)
    width = shared + E * ff
    x = torch.randn(2, K, generator=g, device="cuda").bfloat16()
    w_up = (torch.randn(2 * width, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    w_down = (torch.randn(N, width, generator=g, device="cuda") * 0.1).bfloat16()
    weights = torch.rand(E, generator=g, device="cuda") + 0.1
    kind = dict(act=None, limit=7.0, shared_limit=7.0, alpha=1.702)

    def run(rows, chosen):
        gates = torch.stack([weights * torch.tensor([float(e in c) for e in range(E)], device="cuda") for c in chosen])
        return ops.experts_few(rows, w_up, w_down, gates, None, shared, ff, E, **kind)[0]

    own = set(range(E // 3, E // 3 + top))
    alone = run(x[:1], [own])
    low, high, some = set(range(top)), set(range(E - top, E)), set(range(0, E, E // top))
    for other in (low, high, some, own, set()):
        assert torch.equal(run(x, [own, other])[:1], alone)
        assert torch.equal(run(x.flip(0), [other, own])[1:], alone)
    w_down[:, shared + (E - 1) * ff:] = float("inf")      # of an expert that this token has not chosen
    assert torch.equal(run(x, [own, high])[:1], alone)
