"""Latent attention of single tokens beside a kernel that has started early: its ring's places are read before they are filled again."""

import pytest
import torch

from test_nevurax import _step, dev


def test_producers_of_loaded_rings_have_a_fence():
    """Where a place that warps read by loads is filled again by a bulk copy, a proxy fence stands between the wait and the copy."""
    import os
    import re
    from lite_lang_b200.csrc import build
    for name, wait, copy in (("gemm_stream.cu", r"gt_mbar_wait\(empty0", r"gt_tma_w\("),
                             ("latent_attention_mma.cu", r"at_mbar_wait\(empty0", r"at_tma_3d\(")):
        text = open(os.path.join(build._HERE, name)).read()
        spans = [m.group(0) for m in re.finditer(wait + r"(?:(?!mbar_wait).)*?" + copy, text, re.S)]
        assert spans and all("fence.proxy.async" in s for s in spans), name


@pytest.mark.gpu
@pytest.mark.parametrize("n,T,R,page", [(16, 2048, 512, 16), (16, 4100, 512, 16), (3, 6000, 512, 64), (40, 1500, 384, 16), (5, 3000, 256, 32)])
def test_attention_under_a_kernel_that_started_early(n, T, R, page):
    """Several rounds of the ring and a kernel of many CTAs behind, whose first instructions run on the same SMs: the same bits each time."""
    from lite_lang_b200 import ops
    H, Hd, Hk, d = 12, 12, 2, 128
    assert ops.latent_attention_heads(torch.bfloat16, R, 0) == 16      # (the kernel whose ring this is)
    g = torch.Generator(device=dev())
    g.manual_seed(T + R)
    rnd = dict(generator=g, device=dev())
    q = (0.3 * torch.randn(n, H, R, **rnd)).bfloat16()
    pages = (T + page - 1) // page
    pool = (0.5 * torch.randn(n * pages, 1, page, R, **rnd)).bfloat16()
    table = torch.arange(n * pages, dtype=torch.int32, device=dev()).view(n, -1).contiguous()
    lens = [T - 1 - 37 * i for i in range(n)]
    step = _step([1] * n, lens, list(range(n)))
    splits = ops.latent_attention_splits(n, T)
    # a step of the delta rule behind it (its own inputs)
    off = [0, Hk * d, 2 * Hk * d, 2 * Hk * d + Hd * d]
    proj = torch.randn(n, off[3] + 2 * Hd + Hd * d, **rnd).bfloat16()
    conv = [torch.randn(c, 4, **rnd) for c in (Hk * d, Hk * d, Hd * d)]
    A_log, dt_bias, norm = torch.randn(Hd, **rnd), torch.randn(Hd, **rnd), torch.ones(d, device=dev())
    state = torch.randn(n, Hd * d * d + 3 * (2 * Hk + Hd) * d, **rnd)
    y = torch.empty(n, Hd * d, dtype=torch.bfloat16, device=dev())

    def attend():
        out = torch.empty(n, H, R, dtype=torch.bfloat16, device=dev())
        ops.latent_attention(out, q, pool, table, step, 0, n, H, R, 0, page, None, 0.05, splits, 1)
        return out

    def chain():
        out = attend()
        ops.delta_step(y, proj, *off, proj[:, off[3] + Hd:off[3] + 2 * Hd], None, proj[:, off[3] + 2 * Hd:], None, *conv, A_log, dt_bias,
                       norm, state, Hd * d * d, step, 1e-6, Hd, Hk, d, False, 0)
        return out

    want = attend()
    for i in (0, n - 1):
        rows = pool.view(n, pages * page, R)[i, :lens[i] + 1].double()
        p = torch.softmax(q[i].double() @ rows.t() * 0.05, dim=-1)
        # weights in two bfloat16 terms, float32 sums, one rounding of the result
        assert float((want[i].double() - p @ rows).norm()) <= 2.0 ** -8 * float((p @ rows).norm())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    wrong = 0
    for _ in range(200):
        graph.replay()
        torch.cuda.synchronize()
        wrong += not torch.equal(out, want)
    assert wrong == 0 and int(step.status.item()) == 0
