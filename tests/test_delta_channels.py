"""The delta rule with a decay a key channel by chunks of 64 tokens, beside the recurrence in float64 and the walk by tokens."""

import pytest
import torch

from test_chunk_scan import _LENS, _entry_points, _rel, _step

gpu = pytest.mark.gpu


def test_the_line_of_channels_moves_with_the_heads():
    from lite_lang_b200 import ops
    for heads, low, high in ((2, 250, 320), (12, 192, 256), (24, 96, 128), (28, 80, 128), (48, 48, 64), (112, 16, 32)):
        assert low <= ops.delta_channels_chunked_min(heads, 128, 128) <= high


@gpu
@pytest.mark.parametrize("lens,single,pad", _LENS + [([3, 130] * 17, 0, 5)])
@pytest.mark.parametrize("H,Hk,dk,dv,strong", [(4, 2, 128, 128, 3.0), (3, 3, 64, 128, 60.0), (2, 1, 128, 64, 0.02), (2, 2, 64, 64, 3.0)])
def test_delta_rule_of_channels_by_chunks(lens, single, pad, H, Hk, dk, dv, strong, monkeypatch):
    """strong: the largest exponent of a token's decay; products of a chunk's reach e^-3800, far below float32, and 1."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv + len(lens))
    n, rnd = sum(lens), dict(generator=g, device="cuda")

    def unit(x):
        return x / x.norm(dim=-1, keepdim=True)

    qn = (unit(torch.randn(n, Hk, dk, **rnd)) * dk ** -0.5).reshape(n, -1).contiguous()
    kn = unit(torch.randn(n, Hk, dk, **rnd) + torch.randn(1, Hk, dk, **rnd)).reshape(n, -1).contiguous()
    vc, beta = torch.randn(n, H * dv, **rnd), torch.sigmoid(2 * torch.randn(n, H, **rnd))
    decay = torch.exp(-torch.rand(n, H * dk, **rnd) * torch.linspace(0.01, strong, dk, device="cuda").repeat(H))
    decay[::11, ::3] = 0.0
    slots = list(range(len(lens)))[::-1]
    if pad is not None:
        slots[pad] = -1
    state0 = torch.randn(len(lens) + 1, H * dk * dv + 12, **rnd)
    step, names = _step(lens, slots, single), _entry_points(monkeypatch)
    want, state = torch.zeros(n, H, dv, dtype=torch.float64, device="cuda"), state0.double().clone()
    for e, length in enumerate(lens):
        if slots[e] < 0:
            continue
        a, S = int(step.cu_q[e]), state[slots[e]][:H * dk * dv].view(H, dv, dk).clone()
        q = qn[a:a + length].double().view(length, Hk, dk).repeat_interleave(H // Hk, 1)
        k = kn[a:a + length].double().view(length, Hk, dk).repeat_interleave(H // Hk, 1)
        v = vc[a:a + length].double().view(length, H, dv)
        for t in range(length):
            S = decay[a + t].double().view(H, 1, dk) * S
            u = beta[a + t].double()[:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
            S = S + u[:, :, None] * k[t][:, None, :]
            want[a + t] = (S * q[t][:, None, :]).sum(-1)
        state[slots[e], :H * dk * dv] = S.reshape(-1)
    err = {}
    for way, least in (("walk", 1 << 30), ("chunks", 0)):
        monkeypatch.setattr(ops, "DELTA_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.full((n, H * dv), float("nan"), device="cuda")
        ops.delta_recurrence(qn, kn, vc, beta, decay, st, step, o, H, Hk, dk, dv, True)
        assert int(step.status.item()) == 0
        assert names == ["ll_chunk_delta_scan"] * (way == "chunks") + ["ll_delta_recurrence"] * (way == "walk" or single > 0)
        names.clear()
        assert torch.equal(st[len(lens)], state0[len(lens)])              # a record that no entry names
        if pad == 0:
            assert bool((o == 0).all()) and torch.equal(st, state0)
        else:
            err[way] = (_rel(o.view(n, H, dv), want), _rel(st, state))
    # float32 sums in another order: not above the walk's error (2^-23 where that has hardly any)
    if err:
        assert err["chunks"][0] <= max(err["walk"][0], 2.0 ** -23) and err["chunks"][1] <= max(err["walk"][1], 2.0 ** -23), err


@gpu
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_delta_rule_of_channels_of_numbers_that_are_not_finite(dk, dv, monkeypatch):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv)
    H, lens, rnd = 3, [200, 70], dict(generator=g, device="cuda")
    n = sum(lens)
    qn, kn = (torch.nn.functional.normalize(torch.randn(n, H, dk, **rnd), dim=-1) for _ in range(2))
    vc, beta = torch.randn(n, H, dv, **rnd), torch.rand(n, H, **rnd)
    decay = torch.exp(-torch.rand(n, H * dk, **rnd))
    vc[100, 0, 5], kn[150, 1, 3], vc[30, 2, 40], vc[69 + 200, 2, 0] = float("inf"), float("nan"), float("nan"), -float("inf")
    decay[231, dk + 7] = float("nan")
    state0, step, res = torch.randn(2, H * dk * dv, **rnd), _step(lens, [1, 0]), {}
    for way, least in (("walk", 1 << 30), ("chunks", 0)):
        monkeypatch.setattr(ops, "DELTA_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.empty(n, H * dv, device="cuda")
        ops.delta_recurrence(qn.view(n, -1), kn.view(n, -1), vc.view(n, -1), beta, decay, st, step, o, H, H, dk, dv, True)
        res[way] = (o, st)
    for got, want in zip(res["chunks"], res["walk"]):
        assert bool(torch.isnan(want).any()) and torch.equal(torch.isfinite(got), torch.isfinite(want))
        fin = torch.isfinite(want)
        assert float((got - want)[fin].norm()) <= 1e-5 * float(want[fin].norm())
