"""The delta rule's chunks in parts: what their scratch takes is bounded, and the bits are those of all chunks at once."""

import pytest
import torch

from test_chunk_scan import _entry_points, _step

gpu = pytest.mark.gpu


def _inputs(n, H, Hk, dk, dv, per_channel, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = dict(generator=g, device="cuda")
    unit = lambda: torch.nn.functional.normalize(torch.randn(n, Hk, dk, **rnd), dim=-1).view(n, -1)
    return unit() * dk ** -0.5, unit(), torch.randn(n, H * dv, **rnd), torch.rand(n, H, **rnd), 0.7 + 0.3 * torch.rand(
        n, H * dk if per_channel else H, **rnd)


@gpu
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("lens,single,pad", [([411], 0, None), ([1, 1, 200], 2, None), ([64, 65, 1, 700, 128], 0, 2), ([130] * 34, 0, 5)])
@pytest.mark.parametrize("H,Hk,dk,dv", [(4, 2, 128, 128), (3, 1, 64, 128)])
def test_parts_have_the_bits_of_the_whole(lens, single, pad, H, Hk, dk, dv, per_channel, monkeypatch):
    from lite_lang_b200 import ops
    monkeypatch.setattr(ops, "DELTA_CHUNKED_MIN", 0)
    n, slots = sum(lens), list(range(len(lens)))[::-1]
    if pad is not None:
        slots[pad] = -1
    inputs = _inputs(n, H, Hk, dk, dv, per_channel, n + dk)
    inputs[2][n // 2, 3] = float("inf")
    state0 = torch.randn(len(lens) + 1, H * dk * dv, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    step, names, res = _step(lens, slots, single), _entry_points(monkeypatch), []
    a_chunk = 4 * H * (dv * dk + 64 * dv + 96 * dk + 96 * dk + 64 * 64 + 64 * dk + dk)      # no more than a chunk takes
    for room in (1 << 30, a_chunk, 2 * a_chunk, 5 * a_chunk, 1):
        monkeypatch.setattr(ops, "DELTA_CHUNK_BYTES", room)
        state, o = state0.clone(), torch.full((n, H * dv), 7.0, device="cuda")
        ops.delta_recurrence(*inputs, state, step, o, H, Hk, dk, dv, per_channel)
        assert names[0] == "ll_chunk_delta_scan" and int(step.status) == 0
        names.clear()
        res.append((o.view(torch.int32), state.view(torch.int32)))
    for o, state in res[1:]:
        assert torch.equal(o, res[0][0]) and torch.equal(state, res[0][1])


@gpu
@pytest.mark.parametrize("per_channel", [False, True])
def test_a_long_step_takes_bounded_memory(per_channel):
    from lite_lang_b200 import ops
    H, Hk, d, lens = 28, 4, 128, [5000, 3192]
    inputs = _inputs(sum(lens), H, Hk, d, d, per_channel, 1)
    state, o = torch.zeros(2, H * d * d, device="cuda"), torch.empty(sum(lens), H * d, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    ops.delta_recurrence(*inputs, state, _step(lens, [0, 1]), o, H, Hk, d, d, per_channel)
    assert torch.cuda.max_memory_allocated() - before <= (256 << 20) + (1 << 20)
    assert bool(torch.isfinite(o).all()) and bool(torch.isfinite(state).all())
