"""Two small kernels alone: partial sums that no norm adds up, and the latents' norms beside the cache rows."""

import pytest
import torch

from test_nevurax import dev

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("parts,tokens,n", [(1, 1, 4), (2, 3, 100), (7, 5, 1536), (8, 1, 516), (9, 64, 260), (33, 2, 128)])
def test_partial_sums_are_added_in_their_order(dtype, parts, tokens, n):
    from lite_lang_b200 import ops
    from lite_lang_b200.parts import whole_output
    g = torch.Generator(device="cuda")
    g.manual_seed(parts + n)
    x = torch.randn(parts, tokens, n, generator=g, device="cuda") * torch.logspace(-3, 3, parts, device="cuda")[:, None, None]
    x[0, 0, 1], x[parts - 1, 0, 2], x[0, 0, 3] = float("inf"), float("nan"), -0.0
    want = torch.zeros(tokens, n, device="cuda")
    for p in range(parts):
        want = want + x[p]
    got = ops.sum_parts(x, dtype)
    assert got.dtype == dtype and torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[~got.isnan()], want.to(dtype)[~got.isnan()])
    assert torch.equal(whole_output(x, dtype).nan_to_num(1.0), got.nan_to_num(1.0))


@gpu
def test_partial_sums_of_other_forms():
    """Rows that are no multiple of four numbers, off the boundaries or apart, and other types, are added by the library."""
    from lite_lang_b200 import ops
    from lite_lang_b200.parts import whole_output
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(3, 5, 37, generator=g, device="cuda")
    shifted = torch.empty(3 * 5 * 36 + 1, device="cuda")[1:].view(3, 5, 36).copy_(x[:, :, :36])
    for form in (x, x[:, :, :36], shifted, x.double(), x.to(torch.bfloat16)):
        want = form.double().sum(0)
        assert float((whole_output(form, torch.float32).double() - want).norm() / want.norm()) <= (5e-3 if form.dtype == torch.bfloat16 else 1e-6)
    assert whole_output(torch.empty(2, 0, 8, device="cuda"), torch.bfloat16).shape == (0, 8)
    with pytest.raises(ValueError):
        ops.sum_parts(x.double(), torch.bfloat16)


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [8, 127, 1536, 1537, 2050])          # (1,536 numbers are kept in registers, the rest read twice)
def test_the_queries_latent_has_its_norm_beside_the_cache_rows(dtype, width):
    from lite_lang_b200 import ops
    g = torch.Generator().manual_seed(width)
    H, d, r, R, n, eps = 3, 10, 8, 24, 6, 1e-5
    kv_off = (width + 7) // 8 * 8
    proj = (2.0 * torch.randn(n, kv_off + R + r, generator=g)).to(dtype).to(dev())
    before = proj.clone()
    norm_w, cq_w = (1 + 0.2 * torch.randn(R, generator=g)).to(dev()), (1 + 0.2 * torch.randn(width, generator=g)).to(dev())
    pos = torch.tensor([0, 1, 2, 77, 5, 9], dtype=torch.int32, device=dev())
    slot_map = torch.tensor([9, 3, -1, 0, 17, 12], dtype=torch.int32, device=dev())
    freq = (300.0 ** (-2.0 * torch.arange(r // 2) / r)).float().to(dev())
    status = torch.zeros(1, dtype=torch.int32, device=dev())
    plain, cache = (torch.zeros(5, 1, 4, R + r, dtype=dtype, device=dev()) for _ in range(2))
    q = torch.randn(n, H * (d + r), generator=g).to(dtype).to(dev())
    q_before = q.clone()
    # the cache rows as a call with queries makes them (turned in place), then without queries and with the latent's norm
    ops.latent_prepare(proj, 0, kv_off, norm_w, eps, freq, r, pos, slot_map, plain, None, H, d, r, R, status, q=q, inplace_from=0)
    assert not torch.equal(q, q_before)
    cq = torch.full((n, width), 7.0, dtype=dtype, device=dev())
    ops.latent_prepare(proj, 0, kv_off, norm_w, eps, freq, r, pos, slot_map, cache, None, H, d, r, R, status, inplace_from=0,
                       turn_q=False, cq=cq, cq_norm=cq_w)
    assert torch.equal(cache, plain) and torch.equal(proj, before) and int(status.item()) == 0
    x = before[:, :width].double()
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * cq_w.double()
    tol = 2e-6 if dtype == torch.float32 else 2.0 ** -8          # (one rounding to the type)
    assert float(((cq.double() - want).abs() / want.abs().clamp(min=1e-2)).max()) <= tol
    own = torch.empty_like(cq)
    ops.rmsnorm(own, proj[:, :width], cq_w, eps)
    assert float((cq.double() - own.double()).norm() / own.double().norm()) <= (1e-6 if dtype == torch.float32 else 2e-4)
    # no slots: the norm alone
    cache.zero_()
    cq.fill_(7.0)
    ops.latent_prepare(proj, 0, kv_off, norm_w, eps, freq, r, pos, None, cache, None, H, d, r, R, status, inplace_from=0,
                       turn_q=False, cq=cq, cq_norm=cq_w)
    assert not bool(cache.any()) and float(((cq.double() - want).abs() / want.abs().clamp(min=1e-2)).max()) <= tol
