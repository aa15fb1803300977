"""The delta rule's convolutions over long portions, eight tokens a warp: runs that begin before, at and behind an entry's start,
a padding entry between live ones, heads that fill a warp's accesses and heads that do not, against float64."""

import pytest
import torch

from test_nevurax import _step, dev

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hk,dk,dv,lens", [(3, 1, 128, 64, (301, 1, 2, 259)), (2, 2, 36, 128, (8, 505, 7)),
                                             (2, 1, 132, 20, (512,)), (1, 1, 4, 4, (509, 16))])
def test_runs_of_tokens(dtype, H, Hk, dk, dv, lens):
    from lite_lang_b200 import ops
    g = torch.Generator().manual_seed(dk + len(lens))
    n, Cq, Cv, taps = sum(lens), Hk * dk, H * dv, 4
    C = 2 * Cq + Cv
    ctx = [5 + 3 * i for i in range(len(lens))]
    slots = list(range(len(lens), 0, -1))
    pad = 1 if len(lens) > 2 else None                                  # this entry's record is none
    if pad is not None:
        slots[pad] = -1
    proj = 3.0 * torch.randn(n, C + H, generator=g, dtype=torch.float64)
    proj[n - 20, C - 1], proj[n - 3, C - 2] = float("inf"), -400.0       # beyond the reciprocal's range
    proj, a_in = proj.to(dtype), torch.randn(n, H, generator=g, dtype=torch.float64).to(dtype)
    w = [torch.randn(c, taps, generator=g).abs() + 0.1 for c in (Cq, Cq, Cv)]
    A_log, dt_bias = torch.randn(H, generator=g) - 1.0, torch.randn(H, generator=g)
    tail_off = H * dk * dv
    state = torch.randn(len(lens) + 2, tail_off + (taps - 1) * C, generator=g)
    before = state.clone()
    f32 = dict(dtype=torch.float32, device=dev())
    qn, kn, vc = torch.full((n, Cq), 7.0, **f32), torch.full((n, Cq), 7.0, **f32), torch.full((n, Cv), 7.0, **f32)
    beta, dec, on = torch.empty(n, H, **f32), torch.empty(n, H, **f32), state.to(dev())
    ops.delta_prepare(proj.to(dev()), 0, Cq, 2 * Cq, C, a_in.to(dev()), *(t.to(dev()) for t in w), A_log.to(dev()),
                      dt_bias.to(dev()), on, tail_off, _step(list(lens), ctx, slots), qn, kn, vc, beta, dec, H, Hk, dk, dv, taps, False)
    got = torch.cat([qn, kn, vc], dim=1).double().cpu()
    filt = torch.cat(w).double()
    at = 0
    for e, m in enumerate(lens):
        ours, rows = got[at:at + m], proj[at:at + m, :C].double()
        at += m
        if e == pad:
            assert bool((ours == 7.0).all())
            continue
        old = before[slots[e], tail_off:].double().view(taps - 1, C)     # oldest first
        x = torch.cat([old, rows])
        y = sum(filt[:, j] * x[j:j + m] for j in range(taps))
        # the four products' sum, silu and the root of a unit vector, each in float32: 2^-21 of what the products come to
        bound = 2.0 ** -21 * (1.0 + sum(filt[:, j] * x[j:j + m].abs() for j in range(taps)))
        y = y * torch.sigmoid(y)
        for c0, scale in ((0, dk ** -0.5), (Cq, 1.0)):
            heads, room = y[:, c0:c0 + Cq].view(m, Hk, dk), bound[:, c0:c0 + Cq].view(m, Hk, dk)
            factor = scale / torch.sqrt((heads * heads).sum(-1, keepdim=True) + 1e-6)
            heads *= factor
            room.copy_(2.0 * factor * torch.linalg.vector_norm(room, dim=-1, keepdim=True))
        inf = torch.isinf(y)
        assert torch.equal(inf, torch.isinf(ours)) and bool(((ours - y).abs()[~inf] <= bound[~inf]).all())
        assert torch.equal(on[slots[e], tail_off:].cpu().view(taps - 1, C), x[-(taps - 1):].float())


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_token_has_the_same_bits_in_a_run_and_alone(dtype):
    """A prompt's 600 tokens at once (eight a warp) and in portions of 100 (one a warp)."""
    from lite_lang_b200 import ops
    g = torch.Generator().manual_seed(2)
    n, H, Hk, dk, dv, taps = 600, 4, 2, 128, 128, 4
    Cq, Cv = Hk * dk, H * dv
    C = 2 * Cq + Cv
    proj = (3.0 * torch.randn(n, C + H, generator=g)).to(dtype).to(dev())
    a_in = torch.randn(n, H, generator=g).to(dtype).to(dev())
    w = [torch.randn(c, taps, generator=g).to(dev()) for c in (Cq, Cq, Cv)]
    A_log, dt_bias = torch.randn(H, generator=g).to(dev()), torch.randn(H, generator=g).to(dev())
    tail_off = H * dk * dv

    def made(each):
        state = torch.zeros(2, tail_off + (taps - 1) * C, device=dev())
        outs = []
        for at in range(0, n, each):
            f32 = dict(dtype=torch.float32, device=dev())
            o = [torch.empty(each, c, **f32) for c in (Cq, Cq, Cv, H, H)]
            ops.delta_prepare(proj[at:at + each], 0, Cq, 2 * Cq, C, a_in[at:at + each], *w, A_log, dt_bias, state, tail_off,
                              _step([each], [at], [1]), *o, H, Hk, dk, dv, taps, False)
            outs.append(torch.cat(o, dim=1))
        return torch.cat(outs), state[1, tail_off:].clone()

    (runs, tail), (alone, tail_alone) = made(n), made(100)
    assert torch.equal(runs, alone) and torch.equal(tail, tail_alone)
