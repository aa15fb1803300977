"""The true float32 path on tensor cores: products and prompt attention beside float64 and beside the general kernels."""

import pytest
import torch

gpu = pytest.mark.gpu


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


# rows, features and inner sizes at the edges of tiles (256 x 256), of steps (64) and of parts of k
@gpu
@pytest.mark.parametrize("M,N,K,splits", [(1, 4, 8, 1), (96, 260, 72, 1), (255, 256, 64, 1), (257, 300, 200, 1), (300, 132, 1000, 3),
                                          (513, 1028, 776, 2), (700, 512, 2048, None)])
def test_product(M, N, K, splits):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    wide = torch.randn(M, K + 12, generator=g, device="cuda")
    x = wide[:, 4:4 + K]                                             # rows with a stride of their own
    x[0] *= 1e-20
    w = torch.randn(N, K, generator=g, device="cuda") * torch.logspace(-3, 3, N, device="cuda")[:, None]
    want = x.double() @ w.double().t()
    scale = x.double().abs() @ w.double().abs().t()                  # what a sum's rounding errors are measured by
    got = ops.gemm_f32(x, w, splits=splits)
    # 64 numbers of k a chain of cut-off sums (4 steps of 2^-23), then rounded additions; a term's last bits are 2^-24
    bound = (8 + (K + 63) // 64) * 2.0 ** -24
    assert float(((got.double() - want).abs() / scale.clamp(min=1e-300)).max()) <= bound
    lib = torch.mm(x, w.t())
    assert _rel(got, want) <= max(1.5 * _rel(lib, want), 1.5e-7)
    acc = torch.randn(M, N, generator=g, device="cuda")
    both = acc.double() + want
    ops.gemm_f32(x, w, acc, accumulate=True, splits=splits)
    assert float(((acc.double() - both).abs() / (scale + both.abs())).max()) <= bound + 2.0 ** -23
    parts = ops.gemm_f32(x, w, partial_ok=True, splits=splits)
    assert torch.equal(parts if parts.dim() == 2 else parts.sum(0), got) or _rel(parts.sum(0), got.double()) <= 2e-7


@gpu
@pytest.mark.parametrize("act", ["silu", "relu", "gelu_tanh", "clamped_swish"])
@pytest.mark.parametrize("M,I,K", [(100, 132, 72), (257, 384, 256)])
def test_gated_product(M, I, K, act):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(2 * I, K, generator=g, device="cuda") * K ** -0.5
    kind = ops.GateAct(act, 2.0 if act == "clamped_swish" else 0.0, 1.702)
    got = ops.gemm_f32(x, w, torch.empty(M, I, device="cuda"), gated=kind)
    gu = torch.mm(x.double(), w.double().t())
    want = torch.empty(M, I, device="cuda")
    ops.act_mul(want, gu.float().contiguous(), kind)
    assert float((got - want).abs().max()) <= 4e-6 * float(want.abs().max())


# gate sums that are far out: each beside the same product without a gate and the activation's own kernel, whose sums are the same
# numbers.  Finite inputs whose sums overflow to infinity, gates whose exponential leaves float32, and ordinary ones between them.
@gpu
@pytest.mark.parametrize("act", ["silu", "relu", "gelu_tanh", "clamped_swish"])
def test_gates_that_overflow_and_vanish(act):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    M, I, K = 130, 192, 64
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    x = torch.randn(M, K, generator=g, device="cuda")
    w = torch.randn(2 * I, K, generator=g, device="cuda") * K ** -0.5
    w[:, 1] = 0
    w[:16, 1] = 1e19                                 # sums of 1e39, whose lower terms' products stay finite: +inf in some rows, -inf
    x[:20, 1], x[20:40, 1] = 1e20, -1e20             # in others, beside ordinary ones
    x[40:90, 1:] = 0                                 # one number a row and one a gate: sums of exactly their product, -85 to -105
    x[40:90, 0] = torch.linspace(85, 105, 50, device="cuda")
    w[32:40, 0] = -1.0
    w[40:48, 0] = 1.0
    kind = ops.GateAct(act, 2.0 if act == "clamped_swish" else 0.0, 1.702)
    got = ops.gemm_f32(x, w, torch.empty(M, I, device="cuda"), gated=kind)
    sums = ops.gemm_f32(x, w, splits=1)
    assert bool(torch.isposinf(sums[:20, :16]).all()) and bool(torch.isneginf(sums[20:40, :16]).all())
    want = torch.empty(M, I, device="cuda")
    ops.act_mul(want, sums, kind)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    assert torch.equal(got[want.isfinite()], want[want.isfinite()])


# the epilogue's quotients are the division's: every number of ordinary gates, and of ones spread over the exponential's range
@gpu
@pytest.mark.parametrize("spread", [0.02, 1.0, 30.0])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clamped_swish"])
def test_the_gate_has_the_bits_of_its_own_kernel(act, spread):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x = torch.randn(700, 128, generator=g, device="cuda")
    w = torch.randn(2 * 2048, 128, generator=g, device="cuda") * 128 ** -0.5
    w[:2048] *= spread
    kind = ops.GateAct(act, 7.0 if act == "clamped_swish" else 0.0, 1.702)
    got = ops.gemm_f32(x, w, torch.empty(700, 2048, device="cuda"), gated=kind)
    want = torch.empty(700, 2048, device="cuda")
    ops.act_mul(want, ops.gemm_f32(x, w, splits=1), kind)
    assert torch.equal(got, want)


# more tiles than the device has pairs of blocks: the split terms' buffers go from one tile to the next while both run
@gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("M,N,K", [(701, 17920, 192), (1030, 10248, 136)])
def test_several_tiles_a_pair(M, N, K, gated):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") * K ** -0.5
    want, scale = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    bound = (8 + (K + 63) // 64) * 2.0 ** -24 * scale
    if gated:     # silu(a) * b: a slope of at most 1.1, and a few roundings of the result
        a, b = want.chunk(2, dim=1)
        want = torch.nn.functional.silu(a) * b
        bound = 1.1 * bound[:, :N // 2] * b.abs() + bound[:, N // 2:] * a.abs() + 2.0 ** -21 * want.abs()
    first = None
    for _ in range(5):
        out = torch.empty(M, N // 2 if gated else N, device="cuda")
        got = ops.gemm_f32(x, w, out, **(dict(gated=ops.GateAct("silu")) if gated else dict(splits=1)))
        assert bool(((got.double() - want).abs() <= bound + 1e-12).all())
        assert first is None or torch.equal(first, got)
        first = got.clone()


def test_which_float32_products_go_to_the_tensor_cores():
    from lite_lang_b200 import ops
    x, w = torch.zeros(2048, 1536), torch.zeros(2048, 1536)
    assert not ops.f32_supported(x, w)                               # (not on a CUDA device)


@gpu
@pytest.mark.parametrize("M,N,K,shift,out_pad,taken", [
    (96, 1536, 2048, 0, 0, True), (95, 1536, 2048, 0, 0, False),                # rows
    (256, 512, 2048, 0, 0, True), (256, 508, 2048, 0, 0, False),                # multiply-adds: 2^28
    (96, 64, 65536, 0, 0, True), (96, 60, 65536, 0, 0, False),                  # features
    (300, 1536, 2056, 0, 0, True), (300, 1536, 2052, 0, 0, False),              # numbers of k: a multiple of 8
    (300, 1538, 2048, 0, 0, False),                                             # features: of 4
    (300, 1536, 2048, 1, 0, False), (300, 1536, 2048, 4, 0, True),              # rows that start off 16 bytes
    (300, 1536, 2048, 0, 2, False), (300, 1536, 2048, 0, 4, True),              # outputs of another stride
    (192, 8192, 512, 0, 0, True), (128, 8192, 512, 0, 0, False)])               # few steps of k a tile: the library is faster
def test_dispatch_of_float32_products(M, N, K, shift, out_pad, taken, monkeypatch):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    calls, real = [], ops.gemm_f32
    monkeypatch.setattr(ops, "gemm_f32", lambda *a, **k: (calls.append(k.get("gated")), real(*a, **k))[1])
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K + 8, generator=g, device="cuda")[:, shift:shift + K]
    w = torch.randn(N, K, generator=g, device="cuda")
    want = x.double() @ w.double().t()
    if not out_pad:
        assert _rel(ops.linear(x, w), want) <= 2e-6
        assert bool(calls) == taken
        calls.clear()
    out = torch.empty(M, N + out_pad, device="cuda")[:, :N]
    assert ops.linear(x, w, out) is out and _rel(out, want) <= 2e-6
    assert bool(calls) == taken
    calls.clear()
    acc = torch.randn(M, N + out_pad, generator=g, device="cuda")[:, :N]
    both = acc.double() + want
    ops.linear_accumulate(x, w, acc)
    assert _rel(acc, both) <= 2e-6
    assert bool(calls) == taken


@gpu
@pytest.mark.parametrize("M,I,K,gated", [(1024, 2048, 1024, True), (128, 2048, 1024, False), (300, 1538, 2048, False)])
def test_dispatch_of_gated_float32_products(M, I, K, gated, monkeypatch):
    from lite_lang_b200 import ops
    ops.configure_matmul_precision()
    calls, real = [], ops.gemm_f32
    monkeypatch.setattr(ops, "gemm_f32", lambda *a, **k: (calls.append(k.get("gated")), real(*a, **k))[1])
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(2 * I, K, generator=g, device="cuda") * K ** -0.5
    gu = x.double() @ w.double().t()
    want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    assert _rel(ops.gated_linear(x, w), want) <= 2e-6
    assert any(c is not None for c in calls) is gated


def test_rules_of_float32_products_and_attention():
    """The lines that were measured, both sides (see ops.py)."""
    from lite_lang_b200 import ops
    assert ops.f32_preferred(96, 2048, 1536, 148) and ops.f32_preferred(701, 17920, 1536, 148, True)
    assert ops.f32_preferred(1024, 4096, 1024, 148, True) and not ops.f32_preferred(128, 4096, 1024, 148, True)
    assert not ops.f32_preferred(128, 40000, 72, 148) and ops.f32_preferred(192, 65536, 128, 148)
    assert ops.attn_f32_preferred(64, 2, 64, 148) and ops.attn_f32_preferred(1, 8, 8192, 148)
    assert not ops.attn_f32_preferred(64, 8, 192, 148) and ops.attn_f32_preferred(64, 8, 193, 148)


def test_every_float32_model_loads_the_products_kernel_at_its_start():
    """Whatever its parts are: the first large prompt would build or load it in the middle of a step otherwise."""
    from lite_lang_b200.config import config_from_dict
    from lite_lang_b200.engine.model import CausalLM
    from nevurax_cases import CASES
    for case in CASES.values():
        model = CausalLM(config_from_dict(case["config"]).model_spec())
        model.dtype = torch.float32
        assert "gemm_f32" in model.kernel_libraries()
        model.dtype = torch.bfloat16
        assert "gemm_f32" not in model.kernel_libraries()


@gpu
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nh,nkv,page,window", [(4, 2, 16, None), (6, 1, 5, None), (3, 3, 16, 40), (14, 2, 64, 7)])
def test_prompt_attention(hd, nh, nkv, page, window):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(hd + nh + page)
    spans = [(0, 1), (0, 65), (33, 64), (100, 130), (31, 2)]          # (cached, new) tokens; the first one is not a portion
    pages = [(c + n + page - 1) // page for c, n in spans]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(1)).tolist()
    k = torch.full((sum(pages) + 3, nkv, page, hd), float("nan"), device="cuda")
    v = k.clone()
    table = torch.full((len(spans) + 1, max(pages)), -1, dtype=torch.int32)
    slots, ref = list(range(len(spans)))[::-1], []
    for e, (c, n) in enumerate(spans):
        keys, vals = torch.randn(c + n, nkv, hd, generator=g, device="cuda"), torch.randn(c + n, nkv, hd, generator=g, device="cuda")
        for lp in range(pages[e]):
            table[slots[e], lp] = pg = order.pop()
            rows = slice(lp * page, min((lp + 1) * page, c + n))
            k[pg, :, :rows.stop - rows.start] = keys[rows].transpose(0, 1)
            v[pg, :, :rows.stop - rows.start] = vals[rows].transpose(0, 1)
        ref.append((keys.double(), vals.double()))
    total = sum(n for _, n in spans)
    q = torch.randn(total, nh * hd + 8, generator=g, device="cuda") * 1.5
    ints = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.cumsum(torch.tensor([n for _, n in spans]), 0).tolist(), **ints)
    ctx, slot = torch.tensor([c for c, _ in spans], **ints), torch.tensor(slots, **ints)
    status, table = torch.zeros(1, **ints), table.to("cuda")
    out = torch.full((total, nh * hd), float("nan"), device="cuda")
    ops.attn_f32(out, q, k, v, table, cu[1:], ctx[1:], slot[1:], [n for _, n in spans[1:]], nh, nkv, hd, page, window, hd ** -0.5,
                 status)
    general = torch.empty_like(out)
    req = torch.cat([torch.full((n,), e, **ints) for e, (_, n) in enumerate(spans)])
    pos = torch.cat([torch.arange(c, c + n, **ints) for c, n in spans])
    ops.paged_attention_generic(general, q, q.stride(0), k, v, table, req, slot, pos, total, nh, nkv, hd, page, window,
                                hd ** -0.5, status)
    assert int(status.item()) == 0
    assert bool(torch.isnan(out[0]).all())                            # the token in front is left alone
    want, at = torch.zeros(total, nh, hd, dtype=torch.float64, device="cuda"), 0
    for (c, n), (keys, vals) in zip(spans, ref):
        p, j = torch.arange(c, c + n, device="cuda")[:, None], torch.arange(c + n, device="cuda")[None, :]
        ok = (j <= p) & ((p - j < window) if window else True)
        for h in range(nh):
            s = q[at:at + n, h * hd:(h + 1) * hd].double() @ keys[:, h // (nh // nkv)].t() * hd ** -0.5
            want[at:at + n, h] = torch.softmax(s.masked_fill(~ok, float("-inf")), dim=1) @ vals[:, h // (nh // nkv)]
        at += n
    want = want.view(total, nh * hd)[1:]
    err, was = _rel(out[1:], want), _rel(general[1:], want)
    assert err <= max(1.5 * was, 4e-7), (err, was)


class _Spy:
    """Stands in for the kernel library: what it is called with, and nothing runs."""

    def __init__(self):
        self.status = []

    def call(self, name, *args):
        assert name == "ll_gemm_f32"
        self.status.append(args[-2].value)


def test_products_report_to_the_steps_status_word(monkeypatch):
    """A wait that runs out leaves a wrong output: the kernel has to be handed a word to say so."""
    import threading
    import types

    from lite_lang_b200 import ops
    from lite_lang_b200.engine.model import CausalLM
    spy, word = _Spy(), torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(ops, "_need_cuda", lambda *ts: None)
    monkeypatch.setattr(ops, "load_library", lambda name: spy)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "f32_supported", lambda x, w, **k: x.dtype == torch.float32)
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", False)
    x, w = torch.zeros(96, 64), torch.zeros(64, 64)
    ops.gemm_f32(x, w, status=word)
    assert spy.status.pop() == word.data_ptr()

    def products():
        ops.linear(x, w)
        ops.gated_linear(x, w)
        ops.linear_accumulate(x, w, torch.zeros(96, 64))
        got, spy.status[:] = list(spy.status), []
        return got

    other = []

    def forward(ids, n, status):                       # the model's first part
        other.clear()
        t = threading.Thread(target=lambda: other.extend(products()))
        t.start()
        t.join()
        assert other == [None] * 3                     # (another thread has a step of its own)
        assert products() == [word.data_ptr()] * 3
        return torch.zeros(n, 64)

    model = CausalLM.__new__(CausalLM)
    model.embedding = types.SimpleNamespace(forward=forward)
    model.plan = []
    model.forward(types.SimpleNamespace(num_tokens=96, token_ids=None, status=word, num_logits=0), None)
    assert products() == [None] * 3
    with pytest.raises(RuntimeError), ops.reporting_to(word):
        raise RuntimeError
    assert products() == [None] * 3


def _same_kind(got, want):
    """Finite numbers, NaN and infinities (with their sign) in the same places."""
    return (torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want))
            and torch.equal(torch.isneginf(got), torch.isneginf(want)))


@gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("splits", [1, 3])
def test_product_of_numbers_without_bfloat16_terms(gated, splits):
    """Infinities and numbers above bfloat16's largest: a float32 product keeps them, and every other number stays what it is."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    M, N, K, inf = 300, 264, 520, float("inf")
    x, w = torch.rand(M, K, generator=g, device="cuda") - 0.5, torch.rand(N, K, generator=g, device="cuda") - 0.5
    plain = x.double() @ w.double().t()
    x[3, 500], x[70, 9], x[70, 400], x[290, 1], x[128, 77] = inf, -inf, -inf, 3.4e38, float("nan")
    w[5, 3], w[255, 519], w[130, 64] = -inf, 3.4e38, float("nan")
    w[255] *= 1e-3                                                  # (3.4e35: its sums stay in range, and one term is 3.4e38 x 0)
    x[:, 519], w[255, 519] = x[:, 519] * 1e-3, 3.4e38
    x[290], w[:, 1] = x[290] * 1e-3, w[:, 1] * 1e-3
    x[290, 1] = 3.4e38
    want = (x.double() @ w.double().t()).float()
    bad = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    bad[[3, 70, 290, 128]] = True
    bad[:, [5, 255, 130]] = True
    assert bool(torch.isfinite(want[290]).any()) and bool(torch.isinf(want[3]).any()) and bool(torch.isfinite(want[:, 255]).any())
    if not gated:
        got = ops.gemm_f32(x, w, splits=splits)
        assert _same_kind(got, want)
        fin = torch.isfinite(want)
        scale = x.double().abs() @ w.double().abs().t()
        assert float(((got.double() - want.double()).abs() / scale)[fin].max()) <= (8 + K) * 2.0 ** -24
        return
    if splits != 1:
        return
    for act in ("silu", "relu"):
        got = ops.gemm_f32(x, w, torch.empty(M, N // 2, device="cuda"), gated=ops.GateAct(act))
        ref = torch.empty(M, N // 2, device="cuda")
        ops.act_mul(ref, want.contiguous(), ops.GateAct(act))
        assert _same_kind(got, ref)
        fin = torch.isfinite(ref) & ~bad[:, :N // 2] & ~bad[:, N // 2:]
        assert float((got - ref)[fin].abs().max()) <= 4e-6 * float(ref[fin].abs().max())


@gpu
@pytest.mark.parametrize("hd", [64, 128])
def test_attention_of_numbers_without_bfloat16_terms(hd):
    """A key or value that is not finite shows in the rows that see it, as on the general kernel, and in no other."""
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(hd)
    nh, nkv, page, n, inf = 6, 2, 16, 150, float("inf")
    pages = (n + page - 1) // page
    k, v = (torch.randn(pages, nkv, page, hd, generator=g, device="cuda") for _ in range(2))
    q = torch.randn(n, nh * hd, generator=g, device="cuda")
    ints = dict(dtype=torch.int32, device="cuda")
    table, cu = torch.arange(pages, **ints)[None], torch.tensor([0, n], **ints)
    ctx, slot, status = torch.zeros(1, **ints), torch.zeros(1, **ints), torch.zeros(1, **ints)

    def put(plane, pos, head, channel, value):
        plane[pos // page, head, pos % page, channel] = value

    put(v, 50, 0, 3, inf)
    put(v, 90, 0, 4, 3.4e38)
    put(v, 120, 0, 5, float("nan"))
    put(k, 100, 1, 7, inf)
    put(k, 140, 1, 9, float("nan"))
    q[30, 2] = inf
    for window in (None, 33):
        out, general = torch.empty_like(q), torch.empty_like(q)
        ops.attn_f32(out, q, k, v, table, cu, ctx, slot, [n], nh, nkv, hd, page, window, hd ** -0.5, status)
        ops.paged_attention_generic(general, q, nh * hd, k, v, table, torch.zeros(n, **ints), slot, torch.arange(n, **ints), n, nh,
                                    nkv, hd, page, window, hd ** -0.5, status)
        assert int(status.item()) == 0
        assert _same_kind(out, general)
        assert not bool(torch.isnan(out[:30]).any()) and bool(torch.isinf(out[50]).any())
        fin = torch.isfinite(general) & (general.abs() < 1e30)
        assert float((out - general)[fin].abs().max()) <= 1e-5
        big = torch.isfinite(general) & ~fin
        assert float(((out - general)[big] / general[big]).abs().max()) <= 1e-5


@gpu
@pytest.mark.parametrize("window", [None, 40])
def test_attention_is_the_same_bits_however_a_prompt_is_cut(window):
    from lite_lang_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    nh, nkv, page, n, hd = 6, 2, 16, 200, 64
    pages = (n + page - 1) // page
    k, v = (torch.randn(pages, nkv, page, hd, generator=g, device="cuda") for _ in range(2))
    q = torch.randn(n, nh * hd, generator=g, device="cuda")
    ints = dict(dtype=torch.int32, device="cuda")
    table, slot, status = torch.arange(pages, **ints)[None], torch.zeros(1, **ints), torch.zeros(1, **ints)
    outs = []
    for cuts in ([0, 200], [0, 33, 70, 71, 137, 200]):
        out = torch.empty_like(q)
        for a, b in zip(cuts, cuts[1:]):
            ops.attn_f32(out[a:b], q[a:b], k, v, table, torch.tensor([0, b - a], **ints), torch.tensor([a], **ints), slot, [b - a], nh,
                         nkv, hd, page, window, hd ** -0.5, status)
        outs.append(out)
    assert int(status.item()) == 0
    assert torch.equal(*outs)
