"""What a chunk's decays multiply the state by: their product, rounded once, down to float32's smallest normal numbers."""

import types

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_products_near_the_smallest_numbers(per_channel, dk, dv, monkeypatch):
    """One decay takes the product to 2^-122, the chunk's others leave it above 2^-126; the state is 2^100 in front of it, so that what
    is left of it shows the product's bits.  Keys are zeros: nothing is written."""
    from lite_lang_b200 import ops
    monkeypatch.setattr(ops, "delta_chunked_min", lambda *a: 1)
    monkeypatch.setattr(ops, "delta_channels_chunked_min", lambda *a: 1)
    H, n, scale = 4, 64, 2.0 ** 100
    g = torch.Generator(device="cuda").manual_seed(dk + per_channel)
    rnd = lambda *shape: torch.rand(*shape, generator=g, device="cuda")
    width = H * dk if per_channel else H
    decay = 0.975 + 0.025 * rnd(n, width)
    decay[torch.randint(0, n, (width,), generator=g, device="cuda"), torch.arange(width, device="cuda")] = 2.0 ** -122
    state = torch.full((1, H * dv * dk), scale, device="cuda")
    ints = dict(dtype=torch.int32, device="cuda")
    step = types.SimpleNamespace(cu_q=torch.tensor([0, n], **ints), req_slot=torch.tensor([0], **ints), num_entries=1, num_single=0,
                                 status=torch.zeros(1, **ints))
    q, k = torch.zeros(n, H * dk, device="cuda"), torch.zeros(n, H * dk, device="cuda")
    o = torch.empty(n, H * dv, device="cuda")
    names, real = [], ops.load_library

    def load(name):
        names.append(name)
        return real(name)

    monkeypatch.setattr(ops, "load_library", load)
    ops.delta_recurrence(q, k, rnd(n, H * dv), rnd(n, H), decay, state, step, o, H, H, dk, dv, per_channel)
    assert names == ["chunk_scan"] and int(step.status) == 0
    product = decay.double().prod(0)
    assert float(product.min()) > 2.0 ** -126
    want = product.view(H, 1, -1).expand(H, dv, dk if per_channel else 1).expand(H, dv, dk) * scale
    off = (state.view(H, dv, dk).double() - want).abs() / want
    assert float(off.max()) <= 2.0 ** -24 * (1 + 2.0 ** -20)      # half a unit in the last place: one rounding
