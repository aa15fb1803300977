"""Float32 products of a few tokens on tensor cores: which go there, and their error beside 64 bits."""

import pytest
import torch

gpu = pytest.mark.gpu


def test_which_products_of_few_rows_are_expected_to_gain():
    """Sides of the line that were measured apart (see ops.py)."""
    from lite_lang_b200 import ops
    for m, n, k in ((4, 1536, 8960), (32, 2048, 1536), (40, 1536, 1536), (24, 2048, 11008), (64, 3584, 18944), (20, 3584, 3584)):
        assert ops.f32_preferred(m, n, k, 148)
    for m, n, k in ((4, 1536, 1536), (4, 17920, 1536), (28, 17920, 1536), (8, 37888, 3584), (64, 8192, 512), (64, 512, 512)):
        assert not ops.f32_preferred(m, n, k, 148)


@gpu
@pytest.mark.parametrize("M,N,K,taken", [
    (1, 2048, 11008, False), (2, 2048, 11008, True), (17, 1536, 8960, True), (64, 1536, 8960, True), (65, 1536, 8960, False),
    (40, 2052, 2048, True), (40, 2050, 2048, False), (33, 1020, 4096, False), (33, 1024, 4096, True), (12, 17920, 1536, False)])
def test_products_of_few_rows(M, N, K, taken, monkeypatch):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    calls, real = [], ops.gemm_f32
    monkeypatch.setattr(ops, "gemm_f32", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    want = x.double() @ w.double().t()
    got = ops.linear(x, w)
    assert bool(calls) == taken
    lib = torch.nn.functional.linear(x, w)
    was, err = (float((o.double() - want).norm() / want.norm()) for o in (lib, got))
    # products of all 24 bits and float32 sums: not above the library's error, or a few roundings of 2^-24 where that has few
    assert err <= max(1.05 * was, 2.0 ** -21), (err, was)
    if taken:                                          # under capture, and a row's numbers do not depend on the replay
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            ops.linear(x, w)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            again = ops.linear(x, w)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(again, got)
