"""Products of routed experts on the tensor cores: runs of rows at the edges of tiles, features and inner sizes that no tile
divides, with and without an expert for every token, against float64."""

import pytest
import torch

gpu = pytest.mark.gpu


def _bf16(*shape, gen, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).to(torch.bfloat16)


def _act(name, z):
    if name == "relu2":
        return torch.relu(z) ** 2
    if name == "silu":
        return torch.nn.functional.silu(z)
    return torch.nn.functional.gelu(z, approximate="tanh" if name == "gelu_tanh" else "none")


def _gate(g, u, limit, alpha):
    if limit <= 0:
        return torch.nn.functional.silu(g) * u
    a, c = g.clamp(max=limit), u.clamp(-limit, limit)
    return a * torch.sigmoid(alpha * a) * (c + 1.0)


def _close(got, want):
    """A bfloat16 product, rounded (2^-9 a number), its activation (slopes of a few), rounded again.  All of it, and every row: a
    row of few numbers may have several whose product is rounded the other way (2^-8, and twice that behind a square), and one
    that is small beside the others is held to a part of their mean."""
    want, diff = want.cpu(), got.double().cpu() - want.cpu()
    err = diff.norm() / want.norm()
    assert float(err) <= 0.01, float(err)
    mean = want.norm() / max(1, want.shape[0]) ** 0.5
    rows = diff.norm(dim=-1) / (want.norm(dim=-1) + 0.1 * mean)
    assert float(rows.max()) <= 0.03, float(rows.max())


COUNTS = [(1, 31, 32, 33), (255, 256, 257, 3), (0, 513, 0, 64), (700, 1, 129, 0)]


@gpu
@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("n,k,shared", [(128, 64, (128, 64)), (72, 200, None), (264, 136, (8, 136)), (1000, 512, (520, 512))])
def test_up_and_down_products_of_runs(counts, n, k, shared):
    from lite_lang_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(counts) * 7 + n)
    ends = torch.cumsum(torch.tensor(counts), 0).to(torch.int32).cuda()
    total, E, tokens = sum(counts), len(counts), 300
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rows, row_w = _bf16(total, k, gen=gen), torch.rand(total, generator=gen, device="cuda") + 0.1
    of = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).cuda()
    xs = _bf16(tokens, k + 8, gen=gen)[:, :k] if shared else None            # (rows that are not next to one another)
    shared_w = torch.rand(tokens, generator=gen, device="cuda")
    std = k ** -0.5

    def product(x, w):      # rounded, as the activation reads it
        return (x.double() @ w.double().T).to(torch.bfloat16).double()

    # gated, with clamps and without
    w = _bf16(E, 2 * n, k, gen=gen, std=2 * std)
    ws = _bf16(2 * shared[0], k, gen=gen, std=2 * std) if shared else None
    for limit, limit_s in ((1.5, 2.5), (0.0, 0.0)):
        act = ops.GateAct("clamped_swish", limit, 1.7) if limit else ops.GateAct("silu")
        out, out_s = ops.expert_products(rows, w, ends, True, act, row_w, x=xs, shared=ws, shared_w=shared_w if shared else None,
                                         shared_limit=limit_s, status=status)
        z = torch.stack([product(rows[i:i + 1], w[of[i]])[0] for i in range(total)]) if total < 40 else \
            torch.cat([product(rows[of == e], w[e]) for e in range(E)])
        _close(out, _gate(z[:, :n], z[:, n:], limit, 1.7) * row_w[:, None].double())
        if shared:
            z = product(xs, ws)
            _close(out_s, _gate(z[:, :shared[0]], z[:, shared[0]:], limit_s, 1.7) * shared_w[:, None].double())
    # without a gate
    w = _bf16(E, n, k, gen=gen, std=2 * std)
    ws = _bf16(shared[0], k, gen=gen, std=2 * std) if shared else None
    for name, weight_in in (("relu2", False), ("silu", True), ("gelu_tanh", False), ("gelu", True)):
        out, out_s = ops.expert_products(rows, w, ends, False, name, row_w, weight_in, x=xs, shared=ws, status=status)
        z, rw = torch.cat([product(rows[of == e], w[e]) for e in range(E)]), row_w[:, None].double()
        _close(out, _act(name, z * rw) if weight_in else _act(name, z) * rw)
        if shared:
            _close(out_s, _act(name, product(xs, ws)))
    # the second product: columns of a matrix that holds all experts' one beside the other
    sff = shared[0] if shared else 0
    stacked = _bf16(n, sff + E * k, gen=gen, std=std)
    w = stacked[:, sff:].unflatten(1, (E, k)).permute(1, 0, 2)
    hs = _bf16(tokens, sff, gen=gen) if shared else None
    y, base = ops.expert_products(rows, w, ends, x=hs, shared=stacked[:, :sff] if shared else None, status=status)
    _close(y, torch.cat([rows[of == e].double() @ w[e].double().T for e in range(E)]))
    if shared:
        _close(base, hs.double() @ stacked[:, :sff].double().T)
    assert int(status.item()) == 0


@gpu
@pytest.mark.parametrize("name,weight_in", [("relu2", False), ("silu", True), ("silu", False), ("gelu_tanh", True), ("gelu", False)])
def test_epilogue_without_a_gate_has_the_bits_of_the_activation_kernel(name, weight_in):
    """The product as one without an activation makes it, and the kernel for rows behind it; numbers far out among them."""
    from lite_lang_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    counts, n, k = (700, 3, 0, 321), 520, 512
    ends = torch.cumsum(torch.tensor(counts), 0).to(torch.int32).cuda()
    total = sum(counts)
    rows, w = _bf16(total, k, gen=gen), _bf16(len(counts), n, k, gen=gen, std=4 * k ** -0.5)
    w[0] *= 16.0
    rows[9, 7] = float("-inf")
    row_w = torch.rand(total, generator=gen, device="cuda")
    got, _ = ops.expert_products(rows, w, ends, False, name, row_w, weight_in)
    want, _ = ops.expert_products(rows, w, ends)
    ops.moe_row_act(want, row_w, name, weight_in)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~got.isnan()], want[~want.isnan()])


@gpu
@pytest.mark.parametrize("limit,limit_s", [(0.0, 0.0), (7.0, 3.0)])
def test_gated_epilogue_has_the_bits_of_the_activation_kernel(limit, limit_s):
    """The gate and up products as a product without an activation makes them, and the kernel for rows behind it."""
    from lite_lang_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(8)
    counts, n, k, tokens = (700, 3, 0, 321), 520, 512, 600
    ends = torch.cumsum(torch.tensor(counts), 0).to(torch.int32).cuda()
    total, E = sum(counts), len(counts)
    rows, x = _bf16(total, k, gen=gen), _bf16(tokens, k, gen=gen)
    w, ws = _bf16(E, 2 * n, k, gen=gen, std=4 * k ** -0.5), _bf16(2 * n, k, gen=gen, std=4 * k ** -0.5)
    w[0, :n] *= 8.0                                                      # gates of 30 and more: far into the exponential's range
    x[5, 3], rows[9, 7] = float("inf"), float("-inf")
    row_w, shared_w = torch.rand(total, generator=gen, device="cuda"), torch.rand(tokens, generator=gen, device="cuda")
    act = ops.GateAct("clamped_swish", limit, 1.702) if limit else ops.GateAct("silu")
    out, out_s = ops.expert_products(rows, w, ends, True, act, row_w, x=x, shared=ws, shared_w=shared_w, shared_limit=limit_s)
    z, z_s = ops.expert_products(rows, w, ends, x=x, shared=ws)
    for got, two, weight, lim in ((out, z, row_w, limit), (out_s, z_s, shared_w, limit_s)):
        want = ops.moe_row_gated_act(two, weight, lim, 1.702)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~got.isnan()], want[~want.isnan()])


@gpu
def test_many_groups_and_refusals():
    from lite_lang_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    E, n, k = 256, 16, 64
    ends = (3 * torch.arange(1, E + 1)).to(torch.int32).cuda()
    rows, w = _bf16(3 * E, k, gen=gen), _bf16(E, n, k, gen=gen, std=0.1)
    out, none = ops.expert_products(rows, w, ends)
    assert none is None
    _close(out, torch.einsum("erk,enk->ern", rows.view(E, 3, k).double(), w.double()).reshape(-1, n))
    with pytest.raises(ValueError):
        ops.expert_products(rows.float(), w, ends)
    with pytest.raises(ValueError):
        ops.expert_products(rows, w, ends[:-1].contiguous())
    with pytest.raises(RuntimeError):
        ops.expert_products(rows[:, :60].contiguous(), w[:, :, :60].contiguous(), ends)
