"""How the prefill attention of tcgen05 cuts row blocks: room on the SMs, and no more error with a cut."""
import random

import pytest
import torch

from lite_lang_b200 import ops


def _lengths(entries, group, window, chunk=None, keep=0):
    """Key blocks of 64 of each row block, in order, counted key by key."""
    out, tpb = [], 128 // group
    for ctx, q in entries:
        for first in range(0, q, tpb):
            seen = set()
            for pos in range(ctx + first, ctx + min(first + tpb, q)):
                lo = max(0, pos - window + 1) if window else pos // chunk * chunk if chunk else 0
                seen.update(range(lo // 64, pos // 64 + 1))
            if keep:
                seen.update(range(min((keep + 63) // 64, min(seen))))
            out.append(len(seen))
    return out


@pytest.mark.parametrize("shaped", [False, True])
def test_a_cut_has_room_and_is_shorter(shaped):
    r, cut = random.Random(3 + shaped), 0
    for _ in range(250):
        entries = [(r.choice([0, 0, r.randrange(4000)]), r.randrange(1, 900)) for _ in range(r.randrange(1, 5))]
        group, nkv = r.choice([(1, 12), (6, 2), (7, 4), (8, 2), (16, 1)])
        window, chunk, keep = r.choice([(None, None, 0), (512, None, 0), (300, None, 70 * shaped), (None, 256 if shaped else None, 0)])
        blocks, nsplit, split_len = ops.attn_prefill_tc_plan(entries, group, window, nkv, 296, chunk, keep, shaped=shaped)
        lengths = _lengths(entries, group, window, chunk, keep)
        assert blocks == len(lengths)
        if nsplit == 1:
            assert split_len >= max(lengths)
            continue
        cut += 1
        # what the kernel makes of the plan: even splits, in rounds over the row blocks
        rounds = [0] * nsplit
        longest = 0
        for n in lengths:
            want = min(nsplit, max(1, -(-n // split_len)))
            assert want == -(-n // split_len)               # room for all splits of the longest
            per = -(-n // want)
            longest = max(longest, per)
            for i in range(-(-n // per)):
                rounds[i] += nkv
        last = max(i for i, c in enumerate(rounds) if c)
        assert sum(rounds) <= 296
        assert sum(rounds) + sum(blocks * nkv - c for c in rounds[:last]) <= 296 * 21 // 20 + nkv * blocks * (nsplit > last + 1)
        assert longest < max(lengths) and longest <= split_len
    assert cut > 40


@pytest.mark.gpu
@pytest.mark.parametrize("entries,heads,nkv,window", [
    ([(0, 300)], 12, 2, None), ([(0, 1024)], 12, 2, None), ([(0, 1400)], 12, 2, None), ([(1000, 129), (5, 700)], 16, 2, None),
    ([(4096, 128)], 28, 4, None), ([(0, 409), (0, 682), (0, 957)], 12, 12, 512)])
def test_cut_and_whole_agree(entries, heads, nkv, window):
    page, hd = 16, 128
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    per = [(c + q + page - 1) // page for c, q in entries]
    k, v = (torch.randn(sum(per), nkv, page, hd, generator=g, device="cuda").bfloat16() for _ in range(2))
    table, at = torch.full((len(entries), max(per)), -1, dtype=torch.int32), 0
    for i, n in enumerate(per):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    new = [q for _, q in entries]
    ints = dict(dtype=torch.int32, device="cuda")
    q = torch.randn(sum(new), heads * hd, generator=g, device="cuda").bfloat16()
    cu = torch.tensor([sum(new[:i]) for i in range(len(new) + 1)], **ints)
    outs, status = [], torch.zeros(1, **ints)
    for slots in (0, 2 * ops.sm_count(q.device)):
        blocks, nsplit, split_len = ops.attn_prefill_tc_plan(entries, heads // nkv, window, nkv, slots)
        out = torch.empty_like(q)
        ops.attn_prefill_tc(out, q, q.stride(0), k, v, table.cuda(), cu, torch.tensor([c for c, _ in entries], **ints),
                            torch.arange(len(entries), **ints), len(entries), blocks, heads, nkv, hd, page, window, hd ** -0.5,
                            status, nsplit=nsplit, split_len=split_len)
        outs.append(out.float())
    assert int(status.item()) == 0
    # each against 64 bits.  The cut changes what the sixteen-bit weights are scaled by (the largest score so far) and in what order
    # float32 sums are taken, not how many roundings there are: one of each weight, 2^-9 of it at most, and one of the result; of
    # thousands of independent ones the norms differ by a few parts in a hundred
    want, at, pages = [], 0, 0
    for i, (c, n) in enumerate(entries):
        keys, vals = (t[pages:pages + per[i]].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, :c + n].double()
                      .repeat_interleave(heads // nkv, 0) for t in (k, v))
        rows = q[at:at + n].double().view(n, heads, hd).transpose(0, 1)
        pos, key = torch.arange(c, c + n, device="cuda")[:, None], torch.arange(c + n, device="cuda")[None]
        seen = (key <= pos) & (key > pos - (window or c + n))
        scores = (rows @ keys.transpose(1, 2) * hd ** -0.5).masked_fill(~seen, float("-inf"))
        want.append((scores.softmax(-1) @ vals).transpose(0, 1).reshape(n, -1))
        at, pages = at + n, pages + per[i]
    want = torch.cat(want)
    whole, cut = (float((o.double() - want).norm() / want.norm()) for o in outs)
    assert whole <= 2.0 ** -8 and cut <= 1.1 * whole, (whole, cut)
