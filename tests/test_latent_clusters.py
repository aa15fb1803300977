"""Latent attention of single tokens on tensor cores: every latent width that has straight code or a block size of its own,
pages that come as boxes and pages that do not, rings that wrap, and keys shared out over clusters of every kind of size."""

import math

import numpy as np
import pytest
import torch

from helpers import rel_err
from test_nevurax import _step, dev
from test_rufisun import kernel_tol

gpu = pytest.mark.gpu


@gpu
# R, r: blocks of 64 columns (512, 512 + 64, 256 + 64, 384), of 32 (512 + 32, 256 + 32), of 16 (64 + 16); 1,024: one stage.
# 416, 448, 480: four units of 16 columns a warp, not all of which are there.
# pages of 8 to 128 rows are boxes, of 4 and 12 come row by row.
@pytest.mark.parametrize("H,R,r,page", [(12, 512, 0, 16), (16, 512, 64, 32), (3, 512, 32, 8), (28, 256, 0, 64), (5, 256, 64, 128),
                                        (17, 256, 32, 16), (2, 384, 0, 16), (4, 64, 16, 16), (2, 512, 512, 16), (3, 512, 0, 12),
                                        (4, 160, 32, 4), (2, 416, 0, 16), (3, 416, 32, 12), (12, 448, 0, 16), (2, 448, 64, 32),
                                        (5, 480, 0, 8), (4, 480, 32, 4)])
def test_keys_shared_out_over_clusters(H, R, r, page):
    from lite_lang_b200 import ops
    assert ops.latent_attention_heads(torch.bfloat16, R, r) == 16
    g = torch.Generator().manual_seed(H * 1000 + R + r)
    rng = np.random.default_rng(R)
    KD = R + r
    lens = [1, 64, 65, 130, 700, 449]                         # a tile's edges, and rings that wrap
    rows = [(torch.randn(n, KD, generator=g) * 0.5).to(torch.bfloat16).float() for n in lens]
    q = (torch.randn(len(lens), H, KD, generator=g) * 0.3).to(torch.bfloat16).float()
    pages = [(n + page - 1) // page for n in lens]
    order = rng.permutation(sum(pages) + 3)
    pool = torch.full((sum(pages) + 3, 1, page, KD), float("nan"), dtype=torch.bfloat16)      # (behind the ends, and unowned)
    table = torch.full((len(lens), max(pages)), -1, dtype=torch.int32)
    at = 0
    for i, k in enumerate(rows):
        for j in range(pages[i]):
            table[i, j] = int(order[at])
            part = k[j * page:(j + 1) * page]
            pool[table[i, j], 0, :len(part)] = part.to(torch.bfloat16)
            at += 1
    n = len(lens)
    step = _step([1] * n + [1], [x - 1 for x in lens] + [0], list(range(n)) + [-1])           # (the last one: padding)
    q_dev = torch.cat([q, torch.zeros(1, H, KD)]).to(torch.bfloat16).to(dev()).contiguous()
    sink = torch.randn(H, generator=g) + 1.0
    scale = 1.0 / math.sqrt(KD)
    pool_dev, table_dev = pool.to(dev()), table.to(dev())
    for window, with_sink in ((None, False), (100, True)):
        want = []
        for i, T in enumerate(lens):
            K = rows[i].double()[max(0, T - (window or T)):]
            s = (q[i].double() @ K.T) * scale
            if with_sink:
                s = torch.cat([s, sink.double()[:, None]], dim=1)
            want.append(torch.softmax(s, -1)[:, :len(K)] @ K[:, :R])
        want = torch.stack(want).numpy().reshape(n, -1)
        for nsplit in (1, 2, 3, 6, 9, 16):
            out = torch.full((n + 1, H, R), float("nan"), dtype=torch.bfloat16, device=dev())
            ops.latent_attention(out, q_dev, pool_dev, table_dev, step, 0, n + 1, H, R, r, page, window, scale, nsplit, 1,
                                 sink=sink.to(dev()) if with_sink else None)
            assert int(step.status.item()) == 0
            got = out.float().cpu().numpy().reshape(n + 1, -1)
            assert rel_err(got[:n], want) <= kernel_tol(torch.bfloat16), (window, nsplit)
            assert not got[n].any()


def test_every_latent_width_has_warps_for_all_its_columns():
    from ctypes import c_int
    from lite_lang_b200.ops import load_library
    lib = load_library("latent_attn")
    taken = 0
    for R in range(16, 528, 16):
        for r in range(0, 528, 16):
            if lib.fn("ll_latent_attention_mma_ok")(c_int(R), c_int(r)):
                taken += 1
                columns = lib.fn("ll_latent_attention_mma_columns")(c_int(R), c_int(r))
                assert R <= columns < R + 128, (R, r, columns)
    assert taken > 400


@gpu
def test_a_page_outside_the_pool_sets_the_status_word():
    from lite_lang_b200 import ops
    for page in (16, 12):
        step = _step([1], [40], [0])
        table = torch.tensor([[0, 7, 1, 1]], dtype=torch.int32, device=dev())
        pool = torch.zeros((2, 1, page, 512), dtype=torch.bfloat16, device=dev())
        q = torch.zeros((1, 4, 512), dtype=torch.bfloat16, device=dev())
        ops.latent_attention(torch.empty_like(q), q, pool, table, step, 0, 1, 4, 512, 0, page, None, 0.1, 2, 1)
        assert int(step.status.item()) == 3


@gpu
def test_splits_fit_the_device():
    """All clusters of a plan run at once; a plan has at most a CTA a tile of 64 keys."""
    from lite_lang_b200 import ops
    sms = ops.sm_count(torch.device(dev()))
    for pairs in (1, 5, 16, 40, 64, 100, 200):
        for longest in (10, 300, 9000):
            n = ops.latent_attention_splits(pairs, longest)
            assert 1 <= n <= 16 and n <= (longest + 63) // 64 + 1 and (n == 1 or n * pairs <= sms)


def test_a_plan_belongs_to_its_device(monkeypatch):
    from lite_lang_b200 import ops
    device = [0]

    class Library:
        def fn(self, name):
            return lambda pairs, tiles: 4 + 2 * device[0]

    monkeypatch.setattr(ops, "load_library", lambda name: Library())
    monkeypatch.setattr(torch.cuda, "current_device", lambda: device[0])
    ops._latent_splits.cache_clear()
    try:
        assert ops.latent_attention_splits(3, 1000) == 4
        device[0] = 1
        assert ops.latent_attention_splits(3, 1000) == 6
        device[0] = 0
        assert ops.latent_attention_splits(3, 1000) == 4
    finally:
        ops._latent_splits.cache_clear()


@gpu
def test_threads_that_plan_and_launch_share_a_kernel():
    """One variant of the kernel with rows of 496 and of 1,008 numbers, from two threads on streams of their own, beside plans."""
    import threading
    from lite_lang_b200 import ops
    scale, lens = 0.1, [200, 330]
    step = _step([1, 1], [n - 1 for n in lens], [0, 1])
    table = torch.arange(2 * 21, dtype=torch.int32, device=dev()).view(2, 21)
    g = torch.Generator(device=dev())
    g.manual_seed(2)
    work = []
    for R, r in ((480, 16), (480, 528)):
        q, pool = (torch.randn(*shape, generator=g, device=dev()).to(torch.bfloat16) for shape in ((2, 4, R + r), (42, 1, 16, R + r)))
        want = torch.empty(2, 4, R, dtype=torch.bfloat16, device=dev())
        ops.latent_attention(want, q, pool, table, step, 0, 2, 4, R, r, 16, None, scale, 2, 1)
        work.append((R, r, q, pool, want))
    torch.cuda.synchronize()
    failed = []

    def run(R, r, q, pool, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(300):
                    out = torch.empty_like(want)
                    ops.latent_attention(out, q, pool, table, step, 0, 2, 4, R, r, 16, None, scale, 2, 1)
                    ops._latent_splits.cache_clear()
                    ops.latent_attention_splits(1 + i % 20, 3000)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(out, want)
        except Exception as exc:      # (pytest sees no other thread's)
            failed.append(repr(exc))

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
