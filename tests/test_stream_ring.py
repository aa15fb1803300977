"""The weight-streaming product beside a kernel that has started early: its ring's places are read before they are filled again."""

import pytest
import torch

from test_nevurax import _step, dev


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [9, 12, 16, 24, 32])
@pytest.mark.parametrize("K", [1536, 2048, 3072])
def test_product_under_a_kernel_that_started_early(tokens, K):
    """Rounds of the ring and a kernel of many CTAs behind, whose first instructions run on the same SMs: the same bits each time."""
    from lite_lang_b200 import ops
    H, Hk, d = 16, 2, 128
    off = [0, Hk * d, 2 * Hk * d, 2 * Hk * d + H * d]
    N = off[3] + H + H + H * d
    g = torch.Generator(device=dev())
    g.manual_seed(K + tokens)
    rnd = dict(generator=g, device=dev())
    x, w = torch.randn(tokens, K, **rnd).bfloat16(), (0.03 * torch.randn(N, K, **rnd)).bfloat16()
    conv = [torch.randn(c, 4, **rnd) for c in (Hk * d, Hk * d, H * d)]
    A_log, dt_bias, norm = torch.randn(H, **rnd), torch.randn(H, **rnd), torch.ones(d, device=dev())
    state = torch.randn(tokens, H * d * d + 3 * (2 * Hk + H) * d, **rnd)
    step = _step([1] * tokens, [9] * tokens, list(range(tokens)))
    y = torch.empty(tokens, H * d, dtype=torch.bfloat16, device=dev())
    want = ops.linear(x, w).clone()
    # float32 sums of products of bfloat16: one rounding of the result, and K of the sums
    exact = x.double() @ w.double().t()
    assert float((want.double() - exact).norm()) <= (2.0 ** -9 + K * 2.0 ** -24) * float(exact.norm())

    def chain():
        proj = ops.linear(x, w)
        ops.delta_step(y, proj, *off, proj[:, off[3] + H:off[3] + 2 * H], None, proj[:, off[3] + 2 * H:], None, *conv, A_log, dt_bias,
                       norm, state, H * d * d, step, 1e-6, H, Hk, d, False, 0)
        return proj

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        proj = chain()
    wrong = 0
    for _ in range(200):
        graph.replay()
        torch.cuda.synchronize()
        wrong += not torch.equal(proj, want)
    assert wrong == 0
