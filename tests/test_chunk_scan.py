"""Recurrences of prompt portions by chunks of 64 tokens: beside the recurrence in float64, and which calls go that way."""

import types

import pytest
import torch

gpu = pytest.mark.gpu


def _step(lens, slots, single=0, device="cuda"):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ints = dict(dtype=torch.int32, device=device)
    return types.SimpleNamespace(cu_q=torch.tensor(cu, **ints), req_slot=torch.tensor(slots, **ints),
                                 num_entries=len(lens), num_single=single, status=torch.zeros(1, **ints), lens=lens)


def test_which_portions_go_by_chunks():
    from lite_lang_b200 import ops
    step = _step([1, 1, 100, 156], [0, 1, 2, 3], single=2, device="cpu")
    assert ops.chunked_scan(step, 258, 128, 128, 128) == (2, 2, 256 // 64 + 2)
    assert ops.chunked_scan(step, 258, 128, 128, 129) is None            # too few tokens an entry
    assert ops.chunked_scan(step, 258, 96, 128, 128) is None             # other head sizes stay with the walk
    assert ops.chunked_scan(step, 258, 128, 96, 128) is None
    assert ops.chunked_scan(_step([1, 1], [0, 1], single=2, device="cpu"), 2, 128, 128, 1) is None
    items = ops.chunked_scan(step, 258, 64, 64, 1)[2]
    assert items >= sum((n + 63) // 64 for n in (100, 156))


def test_the_lines_move_with_the_heads():
    """Tokens a portion from which on the chunks were measured ahead (see ops.py): more for few heads, fewer for many."""
    from lite_lang_b200 import ops
    for heads, low, high in ((2, 350, 450), (12, 256, 384), (24, 192, 256), (28, 160, 192), (48, 120, 160), (112, 32, 80)):
        assert low <= ops.decay_chunked_min(heads, 128, 128) <= high
    for heads, low, high in ((2, 200, 260), (12, 160, 256), (24, 96, 128), (28, 96, 128), (48, 56, 80), (112, 16, 48)):
        assert low <= ops.delta_chunked_min(heads, 128, 128) <= high
    assert ops.decay_chunked_min(12, 128, 128) == ops.decay_chunked_min(48, 64, 64)


# lengths at the edges of a chunk, several entries, single tokens in front that stay with the walk, many chunks with a ragged
# end, and (third number) an entry of padding, whose read-outs are zeros
_LENS = [([64], 0, None), ([65, 63, 1, 128], 0, None), ([1, 1, 200], 2, None), ([129, 300], 0, None), ([411], 0, None),
         ([1, 100, 90, 70], 1, 2), ([64], 0, 0)]


def _entry_points(monkeypatch):
    """The names of the kernel libraries' entry points, as they are called."""
    from lite_lang_b200 import ops
    names, real = [], ops.load_library

    class Spy:
        def __init__(self, lib):
            self.lib = lib

        def call(self, name, *args):
            names.append(name)
            return self.lib.call(name, *args)

    monkeypatch.setattr(ops, "load_library", lambda lib: Spy(real(lib)))
    return names


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


@gpu
@pytest.mark.parametrize("lens,single,pad", _LENS)
@pytest.mark.parametrize("dtype,H,hpg,dk,dv,token_decay", [
    (torch.bfloat16, 3, 1, 128, 128, False), (torch.float32, 4, 2, 128, 64, True), (torch.float32, 2, 1, 64, 192, False),
    (torch.bfloat16, 2, 2, 64, 64, True)])
def test_decay_scan_by_chunks(lens, single, pad, dtype, H, hpg, dk, dv, token_decay, monkeypatch):
    """Both ways beside float64: the chunks are no further off than twice the walk's error (float32 sums in another order)."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv + len(lens))
    n, G, rnd = sum(lens), H // hpg, dict(generator=g, device="cuda")
    off = (0, G * dk, 2 * G * dk)
    proj = torch.randn(n, 2 * G * dk + H * dv, **rnd).to(dtype)
    decay = torch.tensor([1 - 2.0 ** (-1 - 3 * i) for i in range(H)], device="cuda")
    td = ts = skip = None
    if token_decay:
        td, ts, skip = torch.exp(-2 * torch.rand(n, H, **rnd)), torch.rand(n, H, **rnd), torch.randn(H, **rnd)
        td[::7] = 0.0                                           # a decay that forgets everything
    slots = list(range(len(lens)))[::-1]
    if pad is not None:
        slots[pad] = -1
    state0 = torch.randn(len(lens) + 1, H * dk * dv, **rnd)
    step, names = _step(lens, slots, single), _entry_points(monkeypatch)
    want, state = torch.zeros(n, H, dv, dtype=torch.float64, device="cuda"), state0.double().clone()
    for e, length in enumerate(lens):
        if slots[e] < 0:
            continue
        a, S = int(step.cu_q[e]), state[slots[e]].view(H, dv, dk).clone()
        rows = proj[a:a + length].double()
        q = rows[:, :G * dk].view(length, G, dk).repeat_interleave(hpg, 1)
        k = rows[:, G * dk:2 * G * dk].view(length, G, dk).repeat_interleave(hpg, 1)
        v = rows[:, 2 * G * dk:].view(length, H, dv)
        for t in range(length):
            d = (td[a + t] if token_decay else decay).double()
            w = ts[a + t].double() if token_decay else torch.ones_like(d)
            S = d[:, None, None] * S + (w[:, None] * v[t])[:, :, None] * k[t][:, None, :]
            want[a + t] = (S * q[t][:, None, :]).sum(-1)
            if token_decay:
                want[a + t] += skip.double()[:, None] * v[t]
        state[slots[e]] = S.reshape(-1)
    err = {}
    for way, least in (("walk", 1 << 30), ("chunks", 1)):
        monkeypatch.setattr(ops, "DECAY_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.full((n, H * dv), float("nan"), device="cuda")
        ops.decay_scan(proj, *off, None if token_decay else decay, st, step, o, H, dk, dv, True, hpg, td, ts, skip)
        assert int(step.status.item()) == 0
        assert names == ["ll_chunk_decay_scan"] * (way == "chunks") + ["ll_decay_scan"] * (way == "walk" or single > 0)
        assert torch.equal(st[len(lens)], state0[len(lens)])          # a record that no entry names
        if pad == 0:
            assert bool((o == 0).all()) and torch.equal(st, state0)
            names.clear()
            continue
        err[way] = (_rel(o.view(n, H, dv), want), _rel(st, state))
        if way == "chunks":
            kept = st.clone()
            ops.decay_scan(proj, *off, None if token_decay else decay, kept, step, o, H, dk, dv, False, hpg, td, ts, skip)
            assert torch.equal(kept, st)                              # not writable: the record stays
        names.clear()
    if pad == 0:
        return
    assert err["chunks"][0] <= max(2 * err["walk"][0], 3e-7) and err["chunks"][1] <= max(2 * err["walk"][1], 3e-7), err


# more entries than a warp has lanes: the walk over chunks then takes them in their order, not by length
@gpu
@pytest.mark.parametrize("lens,single,pad", _LENS + [([3, 130] * 17, 0, 5)])
@pytest.mark.parametrize("H,Hk,dk,dv", [(4, 2, 128, 128), (3, 3, 64, 128), (2, 1, 128, 64), (2, 2, 64, 64)])
def test_delta_rule_by_chunks(lens, single, pad, H, Hk, dk, dv, monkeypatch):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv + len(lens))
    n, rnd = sum(lens), dict(generator=g, device="cuda")

    def unit(x):
        return x / x.norm(dim=-1, keepdim=True)

    qn = (unit(torch.randn(n, Hk, dk, **rnd)) * dk ** -0.5).reshape(n, -1).contiguous()
    kn = unit(torch.randn(n, Hk, dk, **rnd) + torch.randn(1, Hk, dk, **rnd)).reshape(n, -1).contiguous()
    vc, beta = torch.randn(n, H * dv, **rnd), torch.sigmoid(2 * torch.randn(n, H, **rnd))
    decay = torch.exp(-torch.rand(n, H, **rnd) * torch.linspace(0.01, 3.0, H, device="cuda"))
    decay[::11] = 0.0
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
            S = decay[a + t].double()[:, None, None] * S
            u = beta[a + t].double()[:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
            S = S + u[:, :, None] * k[t][:, None, :]
            want[a + t] = (S * q[t][:, None, :]).sum(-1)
        state[slots[e], :H * dk * dv] = S.reshape(-1)
    err = {}
    for way, least in (("walk", 1 << 30), ("chunks", 1)):
        monkeypatch.setattr(ops, "DELTA_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.full((n, H * dv), float("nan"), device="cuda")
        ops.delta_recurrence(qn, kn, vc, beta, decay, st, step, o, H, Hk, dk, dv, False)
        assert int(step.status.item()) == 0
        assert names == ["ll_chunk_delta_scan"] * (way == "chunks") + ["ll_delta_recurrence"] * (way == "walk" or single > 0)
        names.clear()
        if pad == 0:
            assert bool((o == 0).all()) and torch.equal(st, state0)
        else:
            err[way] = (_rel(o.view(n, H, dv), want), _rel(st, state))
    if err:
        assert err["chunks"][0] <= max(2 * err["walk"][0], 3e-7) and err["chunks"][1] <= max(2 * err["walk"][1], 3e-7), err


def _same_kind(got, want):
    return (torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want))
            and torch.equal(torch.isneginf(got), torch.isneginf(want)))


@gpu
@pytest.mark.parametrize("dtype,dk,dv", [(torch.bfloat16, 128, 128), (torch.float32, 128, 64), (torch.float32, 64, 192)])
def test_decay_scan_of_numbers_that_are_not_finite(dtype, dk, dv, monkeypatch):
    """They show from their own token on, in the numbers that the walk by tokens shows them in."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv)
    H, lens, rnd, inf = 3, [200, 70], dict(generator=g, device="cuda"), float("inf")
    n = sum(lens)
    proj = torch.randn(n, H * (2 * dk + dv), **rnd).to(dtype)
    q, k, v = (proj[:, a:b].view(n, H, -1) for a, b in ((0, H * dk), (H * dk, 2 * H * dk), (2 * H * dk, H * (2 * dk + dv))))
    k[100, 0, 5] = inf                      # one channel of a key: every column's read-out
    v[130, 1, 7], v[20, 1, 60] = -inf, float("nan")
    q[40, 2, 3] = inf
    v[235, 2, 1] = 3.4e38 if dtype == torch.float32 else inf
    if dtype == torch.float32:
        k[235, 2] *= 1e-3
    decay, skip = torch.tensor([0.9, 0.99, 1.0], device="cuda"), torch.randn(H, **rnd)
    state0, step, res = torch.randn(2, H * dk * dv, **rnd), _step(lens, [1, 0]), {}
    for way, least in (("walk", 1 << 30), ("chunks", 1)):
        monkeypatch.setattr(ops, "DECAY_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.empty(n, H * dv, device="cuda")
        ops.decay_scan(proj, 0, H * dk, 2 * H * dk, decay, st, step, o, H, dk, dv, True, 1, None, None, skip)
        res[way] = (o, st)
    for got, want in zip(res["chunks"], res["walk"]):
        assert bool(torch.isinf(want).any()) and _same_kind(got, want)
        fin = torch.isfinite(want) & (want.abs() < 1e30)
        assert float((got - want)[fin].norm()) <= 1e-5 * float(want[fin].norm())
    assert int(step.status.item()) == 0


@gpu
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_delta_rule_of_numbers_that_are_not_finite(dk, dv, monkeypatch):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + dv)
    H, lens, rnd = 3, [200, 70], dict(generator=g, device="cuda")
    n = sum(lens)
    qn, kn = (torch.nn.functional.normalize(torch.randn(n, H, dk, **rnd), dim=-1) for _ in range(2))
    vc, beta = torch.randn(n, H, dv, **rnd), torch.rand(n, H, **rnd)
    decay = torch.exp(-torch.rand(n, H, **rnd))
    vc[100, 0, 5], kn[150, 1, 3], vc[30, 2, 40], vc[69 + 200, 2, 0] = float("inf"), float("nan"), float("nan"), -float("inf")
    state0, step, res = torch.randn(2, H * dk * dv, **rnd), _step(lens, [1, 0]), {}
    for way, least in (("walk", 1 << 30), ("chunks", 1)):
        monkeypatch.setattr(ops, "DELTA_CHUNKED_MIN", least)
        st, o = state0.clone(), torch.empty(n, H * dv, device="cuda")
        ops.delta_recurrence(qn.view(n, -1), kn.view(n, -1), vc.view(n, -1), beta, decay, st, step, o, H, H, dk, dv, False)
        res[way] = (o, st)
    for got, want in zip(res["chunks"], res["walk"]):
        assert bool(torch.isnan(want).any()) and torch.equal(torch.isfinite(got), torch.isfinite(want))
        fin = torch.isfinite(want)
        assert float((got - want)[fin].norm()) <= 1e-5 * float(want[fin].norm())
