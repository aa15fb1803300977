"""Plain products of two SMs a tile: every tile width at the edges of rows, columns and k, and SiLU on the first columns."""

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("cols", [0, 128, 192, 256])
@pytest.mark.parametrize("m,n,k", [(65, 8, 8), (256, 192, 64), (257, 193, 72), (300, 520, 136), (1030, 1544, 200)])
def test_tile_widths_and_activated_columns(m, n, k, cols):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda") * 2 * k ** -0.5).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    wide = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    product = x.double() @ w.double().T
    rounded = product.to(torch.bfloat16).double()
    for act_cols in (0, n // 2 + 1, None):
        ops.gemm_pair(x, w, wide[:m, :n], status=status, row_act=None if act_cols == 0 else "silu", act_cols=act_cols, cols=cols)
        first = n if act_cols is None else act_cols
        # (a float32 sum in another order rounds elsewhere now and then: 2^-8 of a number, twice where SiLU follows)
        want = torch.cat([torch.nn.functional.silu(rounded[:, :first]), rounded[:, first:]], dim=1)
        assert float(((wide[:m, :n].double() - want).abs() / (want.abs() + 0.05)).max()) <= 2 ** -6
        assert float((wide[:m, :n].double() - want).norm() / want.norm()) <= 2 ** -8
        assert bool((wide[m:] == 7).all()) and bool((wide[:, n:] == 7).all())
    assert int(status.item()) == 0


def test_columns_of_a_tile():
    from lite_lang_b200 import ops
    for m in (65, 256, 300, 2048, 5000):
        for n in (8, 1536, 6144, 18944):
            assert ops.pair_columns(m, n, 148) in (128, 192, 256)
    assert ops.pair_columns(2048, 6144, 148) == 256 and ops.pair_columns(2048, 1536, 148) == 192


def test_where_silu_goes_into_the_epilogue():
    """Nowhere where it was measured slower (product and kernel, epilogue; us), and where it was faster by a tenth on long ones."""
    from lite_lang_b200 import ops
    for m, n, k, two, one in [(65, 8192, 2048, 9.5, 10.6), (128, 6144, 1536, 8.1, 9.5), (512, 6144, 1536, 12.9, 13.9),
                              (769, 6144, 1536, 18.9, 19.8), (1025, 6144, 1536, 21.7, 23.8), (513, 14336, 3584, 50.0, 61.4),
                              (769, 14336, 3584, 66.4, 79.8), (2048, 1536, 512, 10.0, 10.4), (1280, 3072, 1024, 13.8, 14.1),
                              (1280, 6144, 1536, 26.7, 24.1), (2048, 6144, 1536, 39.5, 31.2), (2049, 14336, 3584, 189.1, 159.0),
                              (8192, 1536, 512, 25.4, 23.5), (2048, 4608, 1024, 24.2, 20.9)]:
        assert ops.silu_preferred(m, n, k) == (one < two), (m, n, k)


@gpu
def test_long_portions_have_silu_in_the_epilogue(monkeypatch):
    from lite_lang_b200 import ops
    calls, real = [], ops.gemm_pair
    monkeypatch.setattr(ops, "gemm_pair", lambda *a, **k: (calls.append(k), real(*a, **k))[1])
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x, w = torch.randn(1030, 1024, generator=g, device="cuda"), torch.randn(4200, 1024, generator=g, device="cuda") / 32
    x, w = x.to(torch.bfloat16), w.to(torch.bfloat16)
    for m, taken in ((1000, True), (300, False), (1030, False)):
        want = (x[:m].double() @ w.double().T).to(x.dtype).double()
        want[:, :3000] = torch.nn.functional.silu(want[:, :3000])
        got = ops.linear_silu(x[:m], w, 3000).double()
        assert float((got - want).norm() / want.norm()) <= 2 ** -7 and bool(calls) == taken
        calls.clear()


@gpu
@pytest.mark.parametrize("dtype,m", [(torch.bfloat16, 300), (torch.bfloat16, 40), (torch.float32, 70)])
def test_product_with_silu_on_its_first_columns(dtype, m):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    x, w = torch.randn(m, 256, generator=g, device="cuda").to(dtype), (torch.randn(200, 256, generator=g, device="cuda") / 8).to(dtype)
    want = (x.double() @ w.double().T).to(dtype).double()
    want[:, :136] = torch.nn.functional.silu(want[:, :136])
    got = ops.linear_silu(x, w, 136).double()
    assert float((got - want).norm() / want.norm()) <= (1e-5 if dtype == torch.float32 else 2 ** -7)


@gpu
@pytest.mark.parametrize("cols", [128, 192, 256])
def test_silu_in_the_epilogue_has_the_bits_of_its_own_kernel(cols):
    """Beside the product alone and the kernel for rows; numbers far out and infinities among them."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    m, n, k, first = 1100, 1544, 256, 1201
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda") * 4 * k ** -0.5).to(torch.bfloat16)
    w[:64] *= 16.0
    x[700, 3], x[701, 3] = float("inf"), float("-inf")
    got, want = (torch.empty(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.gemm_pair(x, w, got, row_act="silu", act_cols=first, cols=cols)
    ops.gemm_pair(x, w, want, cols=cols)
    ops.silu_rows(want[:, :first])
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~got.isnan()], want[~want.isnan()])
