"""The delta rule's single tokens in one launch beside the kernels that make them one by one: the same bits."""

import types

import pytest
import torch

from test_nevurax import _step, dev

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hk,d,per_channel,ranks,gate_act,n,pad", [
    (6, 1, 128, True, (0, 0), 1, 3, 1), (4, 2, 128, False, (0, 0), 0, 5, None), (8, 1, 64, True, (0, 0), 0, 1, None),
    (3, 3, 64, False, (0, 0), 1, 2, 0), (12, 2, 128, True, (64, 64), 1, 2, None), (4, 4, 64, False, (8, 40), 0, 3, 2)])
def test_single_tokens_in_one_launch(dtype, H, Hk, d, per_channel, ranks, gate_act, n, pad):
    from lite_lang_b200 import ops
    if dtype == torch.float32 and ranks == (64, 64):
        ranks = (24, 40)                                                   # (64 and 64 of float32 have no room)
    g = torch.Generator(device=dev())
    g.manual_seed(H * d + n)
    rnd = dict(generator=g, device=dev())
    Cq, Cv, nd = Hk * d, H * d, H * d if per_channel else H
    wide = [ranks[0] or (nd + 7) // 8 * 8, ranks[1] or Cv]
    at, off = 0, []
    for w in (Cq, Cq, Cv, (H + 7) // 8 * 8, *wide):
        off.append(at)
        at += w
    proj = torch.randn(n, at + 8, **rnd).to(dtype)[:, :at]                # a row stride of its own
    w_a = (0.2 * torch.randn(nd, ranks[0], **rnd)).to(dtype) if ranks[0] else None
    w_g = (0.2 * torch.randn(Cv, ranks[1], **rnd)).to(dtype) if ranks[1] else None
    conv = [0.5 * torch.randn(c, 4, **rnd) for c in (Cq, Cq, Cv)]
    A_log, dt_bias, norm = torch.randn(H, **rnd) - 1, torch.randn(nd, **rnd), 1 + 0.1 * torch.randn(d, **rnd)
    tail_off = H * d * d
    first = torch.randn(n + 2, tail_off + 3 * (2 * Cq + Cv), **rnd)
    slots, ctx = list(range(n, 0, -1)), [0, 1, 2, 3, 40][:n]               # records of no, one, two and three inputs
    if pad is not None:
        slots[pad] = -1
    step = _step([1] * n, ctx, slots)
    a_in, gate = proj[:, off[4]:off[4] + (ranks[0] or nd)], proj[:, off[5]:off[5] + (ranks[1] or Cv)]
    got, state = torch.full((n, Cv), float("nan"), dtype=dtype, device=dev()), first.clone()
    assert ops.delta_step_supported(proj, step, H, Hk, d, d, 4, off[:3], w_a, w_g, per_channel, state, tail_off, conv)
    ops.delta_step(got, proj, *off[:4], a_in, w_a, gate, w_g, *conv, A_log, dt_bias, norm, state, tail_off, step, 1e-6, H, Hk, d,
                   per_channel, gate_act)
    # one by one; the ranks' products in float64 (their sum of at most 64 numbers is the one order that differs)
    full = [x if w is None else (x.double() @ w.double().t()).to(dtype) for x, w in ((a_in, w_a), (gate, w_g))]
    f32 = dict(dtype=torch.float32, device=dev())
    qn, kn, vc, beta, dec, o = (torch.empty(n, w, **f32) for w in (Cq, Cq, Cv, H, nd, Cv))
    want, other = torch.empty(n, Cv, dtype=dtype, device=dev()), first.clone()
    ops.delta_prepare(proj, *off[:4], full[0], *conv, A_log, dt_bias, other, tail_off, step, qn, kn, vc, beta, dec, H, Hk, d, d, 4,
                      per_channel)
    ops.delta_recurrence(qn, kn, vc, beta, dec, other, step, o, H, Hk, d, d, per_channel)
    ops.delta_out(want, o, norm, full[1].contiguous(), 1e-6, H, d, gate_act)
    live = [i for i in range(n) if slots[i] >= 0]
    assert torch.equal(state[:, tail_off:], other[:, tail_off:])           # the convolutions' inputs
    if ranks == (0, 0):
        assert torch.equal(state, other) and torch.equal(got[live], want[live])
    else:
        # a rank's number is off by at most one rounding of its storage type (or 2^-20 of float32's sums), 2^-8 of it: a decay
        # by as much of its exponent, of at most 5 here, and a gate by that; everything else is the same
        rel = 2.0 ** -6 if dtype == torch.bfloat16 else 1e-5
        assert float((state - other).norm()) <= rel * float(other.norm())
        assert float((got[live].float() - want[live].float()).norm()) <= rel * float(want[live].float().norm())
    if pad is not None:
        assert bool((got[pad] == 0).all())
    untouched = [i for i in range(n + 2) if i not in slots]
    assert torch.equal(state[untouched], first[untouched])


def test_which_steps_take_one_launch():
    from lite_lang_b200 import ops
    proj, state, conv = torch.zeros(2, 64 * 6 + 8), torch.zeros(3, 2 * 64 * 64 + 3 * 64 * 6), [torch.zeros(128, 4)] * 3
    step = types.SimpleNamespace(num_entries=2)

    def ok(step=step, proj=proj, H=2, Hk=2, dk=64, dv=64, taps=4, off=(0, 64, 128), a=None, g=None, state=state, tail=2 * 64 * 64):
        return ops.delta_step_supported(proj, step, H, Hk, dk, dv, taps, off, a, g, True, state, tail, conv)

    assert ok()
    assert not ok(step=types.SimpleNamespace(num_entries=1))                  # an entry of two tokens
    assert not ok(dv=128) and not ok(dk=32, dv=32) and not ok(taps=3) and not ok(H=9, Hk=1) and not ok(off=(0, 66, 130))
    assert not ok(a=torch.zeros(128, 12)) and not ok(a=torch.zeros(128, 136)) and ok(a=torch.zeros(128, 24))
    assert not ok(proj=torch.zeros(2, 64 * 6 + 7)) and not ok(state=torch.zeros(3, 2 * 64 * 64 + 3 * 64 * 6 + 1))
    assert not ok(a=torch.zeros(128, 128), g=torch.zeros(128, 128))        # no room for the ranks' rows
