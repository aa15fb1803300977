"""Latent attention: keys and values expanded from one cached latent vector per token, sliding window.

Per token the input is projected to ``heads`` queries, each [``dim`` plain | ``rot_dim`` rotated], and to
``kv_rank + rot_dim`` numbers: the first ``kv_rank``, RMS-normed with a weight, are the latent c; the last
``rot_dim`` are one rotated key part shared by all heads.  A head's plain key is Uk_h c, its value Uv_h c;
score = (q_plain . k_plain + q_rot . k_rot) * ``scale``; position i sees j with 0 <= i - j < ``window``
(None: every earlier position); softmax; output projection over the concatenated heads.

Only c and the rotated key part are cached: ``kv_rank + rot_dim`` numbers a token in one plane of a paged
group with one kv head and no value plane.  For single tokens nothing per head is expanded from the cache either: since
q_plain . (Uk_h c) = (Uk_h^T q_plain) . c, the queries are taken into the latent space by a batched product
over heads, attention runs there (keys: the cached rows; values: their first ``kv_rank`` numbers), and a
second batched product expands each head's weighted sum of latents with Uv_h.  That is kv_rank numbers a head, key and
query where the expanded form has ``dim``; portions of prompts, whose queries share the keys, are served with the rows they
see expanded once into every head's keys and values (one product, nothing of it kept) and the tcgen05 attention over them.

Rotation: pairs of the rotated part's first ``rot_dims`` numbers (``rot_layout`` "interleaved": 2i with 2i+1;
"half_split": i with i + rot_dims / 2) turn by position * ``rot_base``^(-2i / rot_dims); the rest passes unchanged.  Angles (float32 position times a
float32 frequency rounded from float64), the latent's norm, scores and softmax are float32.

Further parameters, for designs that differ:
``q_rank``       the queries go through a latent of their own: c_q = RMS norm (weight ``dq.norm``) of W_dq x
                 (``q_rank`` numbers), q = W_uq c_q (tensors ``dq``, ``dq.norm``, ``uq`` in the place of ``q``)
``sink``         every head's softmax has one more key, of the learned score ``sink`` [heads], without a value
``rot_scaling``  (``factor``, ``original``, ``fast``, ``slow``) the slow frequencies stretched and an amplitude on
                 cos and sin, as ``rope_computed`` makes them
``channel_gate`` the heads side by side times sigmoid(W_g x), a gate a channel, x being the input of the projections
                 (tensor ``g`` [heads * vdim, hidden])
"""

from __future__ import annotations

import itertools
from typing import Dict

import torch

from .. import ops
from ..config.spec import PartSpec
from ..config.spec import PartSpec as _PartSpec
from .base import Mixer, PagedKVNeed, TensorDecl, build_part, register_part


class LatentAttention(Mixer):
    def __init__(self, spec: PartSpec):
        super().__init__(spec)
        p = spec.params
        self.hidden_size = int(p["hidden_size"])
        self.H = int(p["heads"])
        self.d = int(p["dim"])
        self.r = int(p["rot_dim"])
        self.dv = int(p["vdim"])
        self.R = int(p["kv_rank"])
        self.window = None if p.get("window") is None else int(p["window"])
        self.scale = float(p.get("scale", (self.d + self.r) ** -0.5))
        self.rot_base = float(p.get("rot_base", 10000.0))
        self.rot_dims = int(p.get("rot_dims", self.r))
        self.eps = float(p["eps"])
        self.q_rank = None if p.get("q_rank") is None else int(p["q_rank"])
        self.sink = bool(p.get("sink", False))
        self.rot_scaling = None if not p.get("rot_scaling") else dict(p["rot_scaling"])
        self.rot_layout = str(p.get("rot_layout", "interleaved"))
        self.channel_gate = bool(p.get("channel_gate", False))
        if self.rot_dims % 2 or not (0 <= self.rot_dims <= self.r):
            raise ValueError("latent_attention: rot_dims must be even and at most rot_dim")
        if self.R > 512:
            raise ValueError("latent_attention: a latent of more than 512 numbers is not built")
        if self.window is not None and self.window <= 0:
            raise ValueError("latent_attention: the window must be positive")
        self.w_in = None
        self.w_uq = self.q_norm_w = self.sink_w = None
        self.amplitude = 1.0

    def tensors(self) -> Dict[str, TensorDecl]:
        h = self.hidden_size
        d: Dict[str, TensorDecl] = {}
        if self.q_rank is None:
            d["q"] = TensorDecl((self.H * (self.d + self.r), h))
        else:
            d["dq"] = TensorDecl((self.q_rank, h))
            d["dq.norm"] = TensorDecl((self.q_rank,), "norm")
            d["uq"] = TensorDecl((self.H * (self.d + self.r), self.q_rank))
        if self.sink:
            d["sink"] = TensorDecl((self.H,), "bias", std=1.0)
        if self.channel_gate:
            d["g"] = TensorDecl((self.H * self.dv, h))
        d.update(self._kv_tensors())
        return d

    def _kv_tensors(self) -> Dict[str, TensorDecl]:
        h = self.hidden_size
        return {
            "dkv": TensorDecl((self.R + self.r, h)),
            "dkv.norm": TensorDecl((self.R,), "norm"),
            "uk": TensorDecl((self.H * self.d, self.R)),
            "uv": TensorDecl((self.H * self.dv, self.R)),
            "o": TensorDecl((h, self.H * self.dv)),
        }

    def load(self, fetch, dtype, device) -> None:
        q = fetch("q" if self.q_rank is None else "dq").to(dtype)
        if self.q_rank is not None:
            self.w_uq = fetch("uq").to(dtype).to(device).contiguous()
            self.q_norm_w = fetch("dq.norm").to(torch.float32).to(device).contiguous()
        if self.sink:
            self.sink_w = fetch("sink").to(torch.float32).to(device).contiguous()
        self.kv_off = (q.shape[0] + 7) // 8 * 8
        rows = [q]
        if self.kv_off != q.shape[0]:
            rows.append(torch.zeros((self.kv_off - q.shape[0], self.hidden_size), dtype=dtype, device=q.device))
        rows.append(fetch("dkv").to(dtype))
        self.gate_off = (self.kv_off + self.R + self.r + 7) // 8 * 8
        if self.channel_gate:
            pad = self.gate_off - self.kv_off - self.R - self.r
            if pad:
                rows.append(torch.zeros((pad, self.hidden_size), dtype=dtype, device=q.device))
            rows.append(fetch("g").to(dtype))
        width = sum(t.shape[0] for t in rows)
        if self.channel_gate and width % 8:      # (rows of the product start on 16-byte boundaries)
            rows.append(torch.zeros((8 - width % 8, self.hidden_size), dtype=dtype, device=q.device))
        self.w_in = torch.cat(rows, dim=0).to(device).contiguous()
        self.norm_w = fetch("dkv.norm").to(torch.float32).to(device).contiguous()
        self.w_uk = fetch("uk").to(dtype).to(device).contiguous().view(self.H, self.d, self.R)
        self.w_uv_t = fetch("uv").to(dtype).to(device).contiguous().view(self.H, self.dv, self.R).transpose(1, 2)
        self.w_o = fetch("o").to(dtype).to(device).contiguous()
        # a cached row into every head's key [plain | rotated] and value: [Uk_h 0; 0 1] for the keys, [Uv_h 0] for the values
        self.w_kv = None
        if dtype == torch.bfloat16 and self.d + self.r == self.dv and self.dv in (64, 128) and (self.R + self.r) % 8 == 0:
            wide = torch.zeros((2, self.H, self.dv, self.R + self.r), dtype=dtype, device=device)
            wide[0, :, :self.d, :self.R] = self.w_uk
            if self.r:
                wide[0, :, self.d:, self.R:] = torch.eye(self.r, dtype=dtype, device=device)
            wide[1, :, :, :self.R] = self.w_uv_t.transpose(1, 2)
            self.w_kv = wide.view(2 * self.H * self.dv, self.R + self.r)
        # frequencies as the rotary part makes them (float64, the scaling's ramp, rounded once)
        rope = build_part("position", _PartSpec("rope_computed", {
            "rotary_dim": self.rot_dims, "theta": self.rot_base, "layout": self.rot_layout,
            "scaling": self.rot_scaling if self.rot_dims else None}))
        self.half_split = not rope.interleaved
        freq = rope.frequencies()
        self.amplitude = float(rope.amplitude)
        self.freq = (freq.to(torch.float32) if freq.numel() else torch.zeros(1)).to(device).contiguous()

    def weight_bytes(self) -> int:
        ts = [self.w_in, self.w_uk, self.w_uv_t, self.w_o, self.w_uq]      # (a step reads these or their expanded form)
        return sum(t.numel() * t.element_size() for t in ts if t is not None)

    def cache_need(self):
        return PagedKVNeed(1, self.R + self.r, self.window, value_head_dim=0)

    def kernel_libraries(self):
        libs = ["core", "latent_attn"]
        if self.w_in is not None and self.w_in.dtype == torch.bfloat16:
            libs.extend(["gemm_smallm", "gemm_stream", "gemm_tc"])
            if self.w_kv is not None:
                libs.append("attn_tc")
        return libs

    # Prompt portions of at least this many tokens go through library products (scores and weighted sums of a
    # block of queries against the run of cached rows they see); shorter ones and single tokens go to the kernel
    # that walks each query's keys itself.
    PRODUCT_MIN_TOKENS = 32
    QUERY_BLOCK = 256
    # Portions of at least this many tokens are served with expanded keys and values, as long as the rows to expand are at
    # most so many times the tokens in them (a row costs (kv_rank + rot_dim) * 2 vdim multiply-adds a head to expand
    # and saves kv_rank * 2 a head and query; below the line the step's time is its launches, which are fewer this way).
    # Measured on a B200, heads of 128, a latent of 512 (in the latent space / this way; us of kernels, us with the host):
    # 12 heads, 2,048 tokens in three requests with a window of 512 237 / 76, 690 / 131; 28 heads, four times 256 behind
    # 2,000 with the window 217 / 85, 361 / 140; one portion of 12 heads: 32 behind 480 33 / 36, 192 / 161, 128 behind 1,920
    # 51 / 54, 187 / 143; 28 heads: 32 behind 480 36 / 42, 186 / 149, 32 behind 1,280 (40 rows a token) 42 / 55, 189 / 152;
    # 2 heads: 128 behind 1,920 35 / 42, 184 / 148.  Where the kernels take a little longer this way, the host decides.
    # Shorter ones stay with the kernel over the latents, which carries the softmax weights in sixteen bits (two terms): the
    # tcgen05 attention has one term of eight, as the products over the latents have.
    EXPAND_MIN_TOKENS = PRODUCT_MIN_TOKENS
    EXPAND_MAX_ROWS = 16
    # Memory that the expanded rows of a call may take at a time: entries are served in groups that stay below it.  (One
    # entry may be more; the products' scores and weights, 6 bytes a head, key and query of a block of 256, are more then.)
    EXPAND_BYTES = 256 << 20

    def _runs(self, step, qrows):
        """How the step's entries are served: (tokens that meet the latents themselves, as runs [(first, behind the last)];
        groups of entries with expanded keys and values [(first entry, their (cached, new) tokens, plan)]).  Layers alike
        share it."""
        key = ("latent_runs", self.H, self.dv, self.R + self.r, self.window)
        if self.w_kv is None or not ops.TC_ENABLED or qrows.stride(0) % 8:
            return [(0, qrows.shape[0])], ()
        got = step.scratch.get(key)
        if got is None:
            got = step.scratch[key] = self._plan_runs(step, qrows)
        return got

    def _plan_runs(self, step, qrows):
        entries = None if getattr(step, "captured", False) else getattr(step, "entries", None)
        ctxs = getattr(step, "entry_ctx", None)
        whole = [(0, qrows.shape[0])], ()
        if entries is None or ctxs is None:
            return whole
        spans = [(c, len(e.tokens)) for c, e in zip(ctxs, entries)]
        long = [(self._seen(c), q) for c, q in spans if q >= self.EXPAND_MIN_TOKENS]
        if not long or sum(c + q for c, q in long) > self.EXPAND_MAX_ROWS * sum(q for _, q in long):
            return whole
        latent, groups, at, e0 = [], [], 0, 0
        for expanded, run in itertools.groupby(spans, lambda span: span[1] >= self.EXPAND_MIN_TOKENS):
            run = list(run)
            if expanded:
                for a, b in self._groups(run):
                    groups.append((e0 + a, run[a:b], ops.attn_prefill_tc_plan(
                        [(self._seen(c), q) for c, q in run[a:b]], 1, self.window, self.H, 2 * ops.sm_count(qrows.device))))
            else:
                latent.append((at, at + sum(q for _, q in run)))
            at += sum(q for _, q in run)
            e0 += len(run)
        return latent, groups

    def _seen(self, ctx: int) -> int:
        """Cached tokens that a portion behind ``ctx`` of them may see."""
        return min(ctx, self.window - 1) if self.window else ctx

    def _groups(self, spans):
        """(first, behind the last) of neighbouring entries whose expanded rows fit ``EXPAND_BYTES`` together."""
        row = 2 * (2 * self.H * self.dv + self.R + self.r)
        first, used = 0, 0
        for i, (c, q) in enumerate(spans):
            need = (self._seen(c) + q + ops.CHUNK - 1) // ops.CHUNK * ops.CHUNK * row
            if i > first and used + need > self.EXPAND_BYTES:
                yield first, i
                first, used = i, 0
            used += need
        yield first, len(spans)

    def _attend_expanded(self, heads, qrows, step, cache, e0, spans, plan) -> None:
        """Entries ``e0`` ... of the step: their ``heads`` rows = attention over expanded keys and values."""
        width, cu_q = self.H * self.dv, step.cu_q[e0:]
        rows, table, rel, own = ops.latent_unpage(cache.k, cache.block_table, cu_q, step.ctx_len[e0:], step.req_slot[e0:], spans,
                                                  self.window, step.status)
        kv = ops.linear(rows, self.w_kv)
        ops.attn_prefill_tc_rows(heads, qrows, kv[:, :width], kv[:, width:], table, cu_q, rel, own, plan, self.H, self.dv,
                                 self.window, self.scale, self.sink_w, step.status)

    def _prepare(self, proj, qrows, step, cache, q_full, front, cq=None) -> None:
        """The new tokens' cache rows and the rotated parts of their queries (``q_full``, in place from token ``front`` on).
        Queries with a latent of their own: the cache rows and that latent's norm ``cq`` first, the rotated parts in a call
        after the second product."""
        second = self.q_rank is not None and cq is None
        ops.latent_prepare(proj, 0, self.kv_off, self.norm_w, self.eps, self.freq, self.rot_dims, step.positions,
                           cache.slot_map if cache.writable and not second else None, cache.k, q_full, self.H, self.d, self.r,
                           self.R, step.status, amplitude=self.amplitude, q=qrows, half_split=self.half_split,
                           inplace_from=0 if cq is not None else front, turn_q=cq is None, cq=cq,
                           cq_norm=None if cq is None else self.q_norm_w)

    def forward(self, x, step, cache):
        n, dev, H, d, r, R = x.shape[0], x.device, self.H, self.d, self.r, self.R
        proj = ops.linear(x, self.w_in)
        qrows = proj
        if self.q_rank is not None:          # the queries' own latent: norm (with the cache rows), then the second product
            cq = torch.empty((n, self.q_rank), dtype=x.dtype, device=dev)
            self._prepare(proj, proj, step, cache, None, 0, cq)
            qrows = ops.linear(cq, self.w_uq)
        latent, groups = self._runs(step, qrows)
        # (tokens in front of the first expanded portion, the step's single tokens among them, have their rotated parts put
        # where the products over heads write; everybody else's are turned where they lie)
        na, front = (latent[-1][1], latent[0][1] if latent[0][0] == 0 else 0) if latent else (0, 0)
        q_full = torch.empty((na, H, R + r), dtype=x.dtype, device=dev) if na else None
        if self.q_rank is None or r:
            self._prepare(proj, qrows, step, cache, q_full, front)
        heads = torch.empty((n, H * self.dv), dtype=x.dtype, device=dev)
        if latent:
            lat = torch.empty((na, H, R), dtype=x.dtype, device=dev)
        for t0, t1 in latent:
            q_head = qrows[t0:t1, :H * (d + r)].view(t1 - t0, H, d + r)
            if t0 >= front and r:
                q_full[t0:t1, :, R:].copy_(q_head[:, :, d:])
            # queries into the latent space: a_h = Uk_h^T q_h, written in front of the rotated parts
            ops.batched_heads(q_head[:, :, :d].permute(1, 0, 2), self.w_uk, out=q_full[t0:t1, :, :R].permute(1, 0, 2))  # [H, tokens, R]
            self.attend(lat, q_full, step, cache, (t0, t1) if groups else None)
            ops.batched_heads(lat[t0:t1].permute(1, 0, 2), self.w_uv_t, out=heads[t0:t1].view(t1 - t0, H, self.dv).permute(1, 0, 2))
        for e0, spans, plan in groups:
            self._attend_expanded(heads, qrows, step, cache, e0, spans, plan)
        if self.channel_gate:
            ops.gate_rows(heads, proj[:, self.gate_off:self.gate_off + H * self.dv])
        return ops.linear(heads, self.w_o, partial_ok=self.partial_ok)

    def _splits(self, n, step, device):
        """(CTAs that share a query's keys, tiles of 32 positions each takes).  On tensor cores a CTA has 16 of a query's heads
        and the CTAs that share its keys are a cluster (``ops.latent_attention_splits``), which shares out the query's own
        tiles.  On the other kernel a CTA has 8 heads, few queries (decode steps) are spread until the CTAs fill the device
        about twice (a tile is a chain of latencies), and the plan is made for the longest run of keys any query of the step
        may see (a captured step: of its class of context lengths)."""
        longest = step.max_kv_len if self.window is None else min(step.max_kv_len, self.window)
        tiles = (longest + 31) // 32 + 1                       # (a run that starts inside a tile touches one more)
        group = ops.latent_attention_heads(self.w_o.dtype, self.R, self.r)
        ctas = n * ((self.H + group - 1) // group)
        if group == 16:
            nsplit = ops.latent_attention_splits(ctas, longest)
        else:
            nsplit = max(1, min(tiles, (2 * ops.sm_count(device)) // max(1, ctas), 16))
        return nsplit, (tiles + nsplit - 1) // nsplit

    def attend(self, lat, q_full, step, cache, tokens=None) -> None:
        """All of the step's tokens, or (``tokens``) a run of single tokens and short portions."""
        n, H, R, r = q_full.shape[0], self.H, self.R, self.r
        args = (H, R, r, cache.page_size, self.window, self.scale)
        entries = None if getattr(step, "captured", False) else getattr(step, "entries", None)
        if tokens is not None or entries is None or all(len(e.tokens) < self.PRODUCT_MIN_TOKENS for e in entries):
            t0, t1 = tokens or (0, n)
            ops.latent_attention(lat, q_full, cache.k, cache.block_table, step, t0, t1 - t0, *args,
                                 *self._splits(t1 - t0, step, lat.device), sink=self.sink_w)
            return
        t, run0 = 0, 0          # run0: first token of the current run of entries that go to the kernel
        for e, ctx in zip(entries, step.entry_ctx):
            q = len(e.tokens)
            if q >= self.PRODUCT_MIN_TOKENS:
                if t > run0:
                    ops.latent_attention(lat, q_full, cache.k, cache.block_table, step, run0, t - run0, *args,
                                         sink=self.sink_w)
                self._attend_by_products(lat, q_full, cache, step, e.slot, t, q, ctx)
                run0 = t + q
            t += q
        if n > run0:     # (padding entries of a captured step never come here: such a step has no host entries)
            ops.latent_attention(lat, q_full, cache.k, cache.block_table, step, run0, n - run0, *args,
                                 sink=self.sink_w)

    def _attend_by_products(self, lat, q_full, cache, step, slot, t0, count, ctx) -> None:
        """Tokens t0 .. t0 + count - 1 of the step: one request's positions ctx .. ctx + count - 1."""
        H, R, KD = self.H, self.R, self.R + self.r
        for b0 in range(0, count, self.QUERY_BLOCK):
            nb = min(self.QUERY_BLOCK, count - b0)
            p0 = ctx + b0
            first = max(0, p0 - self.window + 1) if self.window else 0
            # the run starts at a multiple of 8 positions and is 8 k rows long (zero rows around the cached ones):
            # widths that the library's fast kernels take
            lo = first // 8 * 8
            keys = torch.empty(((p0 + nb - lo + 7) // 8 * 8, KD), dtype=lat.dtype, device=lat.device)
            ops.latent_gather(keys, cache.k, cache.block_table, slot, lo, cache.page_size, step.status,
                              first=first, last=p0 + nb - 1)
            qb = q_full[t0 + b0:t0 + b0 + nb].view(nb * H, KD)
            scores = ops.linear(qb, keys, out_dtype=torch.float32, weight_made=True)     # [nb * H, keys]
            weights = torch.empty(scores.shape, dtype=lat.dtype, device=lat.device)
            ops.latent_masked_softmax(weights, scores, H, p0, lo, self.window, self.scale, sink=self.sink_w)
            ops.product(weights, keys[:, :R], out=lat[t0 + b0:t0 + b0 + nb].view(nb * H, R))


register_part("mixer", "latent_attention", LatentAttention)
