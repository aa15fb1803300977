"""Linear attention's and retention's single tokens in one launch beside the kernels that make them one by one: the same bits."""

import types

import pytest
import torch

from test_nevurax import _step, dev

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,n,pad,kind,rot,interleaved,writable", [
    (3, 128, 5, 1, "silu", 0, True, True), (2, 64, 2, None, "silu", 0, True, False), (3, 128, 3, 0, "turned", 128, False, True),
    (2, 64, 4, None, "turned", 64, False, True), (2, 128, 2, None, "turned", 36, True, True), (2, 64, 1, None, "turned", 16, True, False),
    (1, 128, 2, None, "turned", 0, True, True), (2, 128, 3, 2, "turned", 40, False, True)])
def test_single_tokens_in_one_launch(dtype, H, d, n, pad, kind, rot, interleaved, writable):
    from lite_lang_b200 import ops
    g = torch.Generator(device=dev())
    g.manual_seed(H * d + n + rot)
    rnd = dict(generator=g, device=dev())
    C = H * d
    proj = torch.randn(n, 4 * C + 8, **rnd).to(dtype)[:, :4 * C]           # a row stride of its own
    at, gate = (0, C, 2 * C), proj[:, 3 * C:]
    decay, freq = torch.rand(H, **rnd), torch.rand(rot // 2, **rnd) if rot else None
    first = torch.randn(n + 2, C * d + 4, **rnd)
    slots = list(range(n, 0, -1))
    if pad is not None:
        slots[pad] = -1
    step = _step([1] * n, [0, 1, 700, 5000, 3][:n], slots)
    assert ops.decay_step_supported(proj, at, step, H, d, d, first, rot, interleaved)
    f32 = dict(dtype=torch.float32, device=dev())
    state, other, o = first.clone(), first.clone(), torch.full((n, C), float("nan"), **f32)
    if kind == "silu":
        got = torch.full((n, C), float("nan"), **f32)
        ops.decay_step(proj, at, decay, state, step, H, d, o=got, silu=True, write_state=writable)
        rows = proj[:, :3 * C].contiguous()
        ops.silu_rows(rows)
        ops.decay_scan(rows, *at, decay, other, step, o, H, d, d, writable)
        want = o
    else:
        got, want = torch.full((n, C), float("nan"), dtype=dtype, device=dev()), torch.empty(n, C, dtype=dtype, device=dev())
        ops.decay_step(proj, at, decay, state, step, H, d, y=got, gate=gate, eps=1e-5, freq=freq, interleaved=interleaved,
                       k_scale=d ** -0.5, write_state=writable)
        rows = torch.empty(n, 3 * C, **f32)
        ops.rotate_rows_f32(rows, at, proj, at, step.positions, freq, interleaved, H, d, C, 1.0, d ** -0.5)
        ops.decay_scan(rows, *at, decay, other, step, o, H, d, d, writable)
        ops.head_norm_gate_out(want, o, gate, 1e-5, H, d, "silu")
    assert int(step.status.item()) == 0
    live = [i for i in range(n) if slots[i] >= 0]
    assert torch.equal(state, other) and torch.equal(got[live], want[live])
    assert writable or torch.equal(state, first)
    if pad is not None:
        assert bool((got[pad] == 0).all())


def test_which_steps_take_one_launch():
    from lite_lang_b200 import ops
    step, state = types.SimpleNamespace(num_entries=2), torch.zeros(3, 2 * 64 * 64)

    def ok(proj=torch.zeros(2, 512), at=(0, 128, 256), step=step, dk=64, dv=64, state=state, **k):
        return ops.decay_step_supported(proj, at, step, 2, dk, dv, state, **k)

    assert ok() and ok(rot=64, interleaved=False) and ok(rot=36)
    assert not ok(step=types.SimpleNamespace(num_entries=1)) and not ok(dv=128) and not ok(dk=32, dv=32) and not ok(at=(0, 130, 260))
    assert not ok(proj=torch.zeros(2, 514)) and not ok(state=torch.zeros(3, 2 * 64 * 64 + 2)) and not ok(rot=36, interleaved=False)
    assert not ok(rot=66) and not ok(rot=128)
