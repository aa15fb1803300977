"""What the speed of this engine is measured on.

The cases are what a server built on the engine runs: whole steps of a Qwen2 model through ``ModelRunner.step`` (decode
and prompt, bfloat16 and float32), and single parts of the other designs' layers through the parts' own interface
(``build_part`` ... ``forward``): routed experts, the gated delta rule, linear attention with decay, retention, latent
attention and attention with shaped scores, each for prompt portions and for single tokens.  Parts that serve single
tokens are captured in a CUDA graph and replayed, as the runner does with a step of single tokens.

Sizes are those of the benchmark: Qwen2 1.5B, 2.5-3B and 7B, and layers of the other designs as large as those.
"""

from __future__ import annotations

import math

import torch

DEV = "cuda"
PAGE = 16

# width, heads, kv heads, inner width of the feed-forward, experts and how many of them a token uses, window
SIZES = {
    "1p5b": dict(width=1536, heads=12, kv=2, inter=8960, experts=16, top=4, window=512),
    "3b": dict(width=2048, heads=16, kv=2, inter=11008, experts=16, top=4, window=512),
    "7b": dict(width=3584, heads=28, kv=4, inter=18944, experts=8, top=2, window=1024),
}
HEAD = 128
VOCAB = 151936
ALPHA, LIMIT = 1.702, 7.0          # the gated experts' clamped swish
BIAS_ROWS, KEEP_FIRST = 32, 64     # the shaped attention's distance table, and the first tokens that stay visible


def listed():
    return [
        # generation for eight users at once: the benchmark's own step
        dict(name="qwen2_decode_b8", kind="qwen2", mode="decode", size="1p5b", layers=28, batch=8, context=2048,
             dtype="bfloat16"),
        # a busy server: 64 requests, half of the bytes are the cache
        dict(name="qwen2_decode_b64", kind="qwen2", mode="decode", size="1p5b", layers=28, batch=64, context=2048,
             dtype="bfloat16"),
        # a long prompt's first token
        dict(name="qwen2_prefill_2048", kind="qwen2", mode="prefill", size="1p5b", layers=28, batch=1, tokens=2048,
             dtype="bfloat16"),
        # the true 32-bit path, two prompts of odd lengths in one step (layers of the same size; four of them)
        dict(name="qwen2_f32_prefill", kind="qwen2", mode="prefill", size="1p5b", layers=4, batch=2, tokens=701,
             dtype="float32"),
        # routed feed-forward of a prompt portion: gated experts, a shared one with a gate
        dict(name="experts_prefill", kind="experts", mode="prefill", size="1p5b", design="gated", tokens=2048),
        # the same part for eight single tokens: squared-relu experts, all of them are read
        dict(name="experts_decode_b8", kind="experts", mode="decode", size="1p5b", design="relu2", batch=8),
        # gated delta rule: two prompts of odd lengths in a step
        dict(name="delta_prefill", kind="delta", mode="prefill", size="1p5b", design="head", batch=2, tokens=2047),
        # one user's next token: the smallest call there is
        dict(name="delta_decode_b1", kind="delta", mode="decode", size="1p5b", design="channel", batch=1, context=64),
        # linear attention with decay, a whole portion of one prompt
        dict(name="linear_prefill", kind="linear", mode="prefill", size="1p5b", design="linear", batch=1, tokens=2048),
        # latent attention with a window: a prompt portion of three requests
        dict(name="latent_prefill", kind="latent", mode="prefill", size="1p5b", design="window", batch=3, tokens=2048),
        # latent attention over the whole context for sixteen single tokens
        dict(name="latent_decode_b16", kind="latent", mode="decode", size="1p5b", design="full", batch=16,
             context=2048),
        # windowed attention with a distance bias, kept first tokens, a learned sink and a gate a channel
        dict(name="shaped_prefill", kind="shaped", mode="prefill", size="7b", batch=2, tokens=1500),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["qwen2", "qwen2", "qwen2", "experts", "experts", "delta", "delta", "linear", "linear", "latent",
                       "latent", "shaped"])
    mode = rng.choice(["prefill", "decode"])
    size = rng.choice(["1p5b", "1p5b", "3b", "7b"])
    if kind == "qwen2":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        if mode == "decode":
            return dict(kind=kind, mode=mode, size=size, layers=4, batch=_spread(rng, 1, 64),
                        context=_spread(rng, 128, 4096), dtype=dtype)
        tokens = _spread(rng, 64, 2048 if dtype == "bfloat16" else 700)
        return dict(kind=kind, mode=mode, size=size, layers=4, batch=min(rng.randint(1, 4), tokens // 16),
                    tokens=tokens, dtype=dtype)
    case = dict(kind=kind, mode=mode, size=size)
    if kind == "experts":
        case["design"] = rng.choice(["relu2", "gated"])
    elif kind == "delta":
        case["design"] = rng.choice(["head", "channel"])
    elif kind == "linear":
        case["design"] = rng.choice(["linear", "retention"])
    elif kind == "latent":
        case["design"] = rng.choice(["window", "full"])
    if mode == "prefill":
        case["tokens"] = _spread(rng, 64, 2048)
        if kind != "experts":
            case["batch"] = min(rng.randint(1, 4), case["tokens"] // 16)
    else:
        case["batch"] = _spread(rng, 1, 64)
        if kind != "experts":
            case["context"] = _spread(rng, 128, 4096)
    return case


# ---------------------------------------------------------------------------------------------------------
# inputs: everything from the seed, on the device
# ---------------------------------------------------------------------------------------------------------
def _gen(seed, part):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + part) % (1 << 62))
    return g


def _normal(g, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    """Numbers that checkpoints hold: bfloat16, or bfloat16-rounded float32."""
    t = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(mean, std, generator=g).to(torch.bfloat16)
    return t if dtype == torch.bfloat16 else t.to(dtype)


def _dims(case):
    d = dict(SIZES[case["size"]])
    d["vocab"] = VOCAB if case.get("layers") == 28 else 32768
    top, inter = d["top"], d["inter"]
    # as many active weights as the dense feed-forward has
    d["ff"] = (inter if case.get("design") == "gated" else 3 * inter // 2) // (top + 1) // 64 * 64
    d["rank"] = 4 * HEAD
    d["q_rank"] = 3 * d["width"] // 4 // 64 * 64
    return d


def _lengths(case):
    """Tokens of each request of a prompt portion: unequal shares, together ``tokens``."""
    n, b = case["tokens"], case.get("batch", 1)
    weights = [3 + 2 * ((i * 5) % 4) for i in range(b)]
    shares = [max(1, n * w // sum(weights)) for w in weights]
    shares[-1] += n - sum(shares)
    return shares


def _contexts(case):
    """Cached tokens of each request of a decode step, between half of ``context`` and all of it."""
    c = case["context"]
    return [c - (i * 37) % max(1, c // 2) for i in range(case["batch"])]


def _weights(case, seed):
    """The tensors of a checkpoint, by name."""
    g, d = _gen(seed, 1), _dims(case)
    w, h, kv, kind = d["width"], d["heads"], d["kv"], case["kind"]
    out = {}

    def mat(name, rows, cols, std=0.02):
        out[name] = _normal(g, (rows, cols), std)

    def vec(name, n, std, mean=0.0):
        out[name] = _normal(g, (n,) if isinstance(n, int) else n, std, mean)

    if kind == "qwen2":
        # the matrices that write into the residual stream are smaller, the deeper the model, as such models are
        # initialised, and the stream is not all layers' output: roundings of one layer then stay as small in the next
        mat("model.embed_tokens.weight", d["vocab"], w, 0.5)
        small = 0.02 / math.sqrt(2 * case["layers"])
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", w, 0.05, 1.0)
            vec(p + "post_attention_layernorm.weight", w, 0.05, 1.0)
            for n, rows in (("q", h * HEAD), ("k", kv * HEAD), ("v", kv * HEAD)):
                mat(p + f"self_attn.{n}_proj.weight", rows, w)
                vec(p + f"self_attn.{n}_proj.bias", rows, 0.02)
            mat(p + "self_attn.o_proj.weight", w, h * HEAD, small)
            mat(p + "mlp.gate_proj.weight", d["inter"], w)
            mat(p + "mlp.up_proj.weight", d["inter"], w)
            mat(p + "mlp.down_proj.weight", w, d["inter"], small)
        vec("model.norm.weight", w, 0.05, 1.0)
    elif kind == "experts":
        gated = case["design"] == "gated"
        mat("router", d["experts"], w, 0.03)
        if gated:
            vec("router.b", d["experts"], 0.3)
            mat("shared.sg", 1, w, 0.03)
        for name in [f"e{e}" for e in range(d["experts"])] + ["shared"]:
            if gated:
                mat(name + ".gate", d["ff"], w)
            mat(name + ".up", d["ff"], w)
            mat(name + ".down", w, d["ff"])
    elif kind == "delta":
        cq, cv = kv * HEAD, h * HEAD
        for name, rows in (("q", cq), ("k", cq), ("v", cv)):
            mat(name, rows, w)
            vec(name + ".conv", (rows, 4), 0.4)
        mat("b", h, w)
        vec("A_log", h, 0.5, -1.0)
        vec("norm", HEAD, 0.05, 1.0)
        mat("o", w, cv)
        if case["design"] == "channel":
            vec("dt_bias", h * HEAD, 0.5)
            mat("a1", 64, w)
            mat("a2", h * HEAD, 64, 0.1)
            mat("g1", 64, w)
            mat("g2", cv, 64, 0.1)
        else:
            vec("dt_bias", h, 0.5)
            mat("a", h, w)
            mat("g", cv, w)
    elif kind == "linear":
        for name in ("q", "k", "v", "g"):
            mat(name, h * HEAD, w)
        mat("o", w, h * HEAD)
        if case["design"] == "linear":
            vec("norm", h * HEAD, 0.05, 1.0)
    elif kind == "latent":
        if case["design"] == "window":
            mat("q", h * HEAD, w)
        else:
            mat("dq", d["q_rank"], w)
            vec("dq.norm", d["q_rank"], 0.05, 1.0)
            mat("uq", h * HEAD, d["q_rank"])
        mat("dkv", d["rank"] + _rot(case), w)
        vec("dkv.norm", d["rank"], 0.05, 1.0)
        mat("uk", h * (HEAD - _rot(case)), d["rank"], 0.04)
        mat("uv", h * HEAD, d["rank"], 0.04)
        mat("o", w, h * HEAD)
    else:
        for name, rows in (("q", h * HEAD), ("k", kv * HEAD), ("v", kv * HEAD), ("g", h * HEAD)):
            mat(name, rows, w)
        mat("o", w, h * HEAD)
        vec("sink", h, 1.0)
        vec("rel", (BIAS_ROWS, h), 0.5)
    return out


def _rot(case):
    return 32 if case["design"] == "window" else 0


def _decays(heads):
    return [1.0 - 2.0 ** (-2 - 6 * i / max(heads - 1, 1)) for i in range(heads)]


def _rows(case, seed):
    """What a part reads: a norm's output, a row a token."""
    n = case["tokens"] if case["mode"] == "prefill" else case["batch"]
    return _normal(_gen(seed, 2), (n, _dims(case)["width"]))


def _cached(case, seed):
    """What a decode step finds in the cache, by plane and request: (keys, values or None), or the state records."""
    d, g = _dims(case), _gen(seed, 3)
    kind, kv = case["kind"], d["kv"]
    dtype = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    if kind in ("delta", "linear"):
        shape = (case["batch"], d["heads"], HEAD, HEAD)            # [request, head, value column, key channel]
        state = torch.empty(shape, device=DEV).normal_(0.0, 0.3, generator=g)
        if kind == "delta":
            taps = torch.empty((case["batch"], 3, (2 * kv + d["heads"]) * HEAD), device=DEV).normal_(0, 0.8, generator=g)
            return state, taps
        return state, None
    longest = max(_contexts(case))
    if kind == "latent":
        shape, value = (1, case["batch"], longest, 1, d["rank"] + _rot(case)), False
    else:
        shape, value = (case.get("layers", 1), case["batch"], longest, kv, HEAD), True
    k = torch.stack([_normal(g, shape[1:], 0.8, dtype=dtype) for _ in range(shape[0])])
    v = torch.stack([_normal(g, shape[1:], 0.8, dtype=dtype) for _ in range(shape[0])]) if value else None
    return k, v


def _tokens(case, seed):
    n = case["tokens"] if case["mode"] == "prefill" else case["batch"]
    return torch.randint(0, _dims(case)["vocab"], (n,), generator=_gen(seed, 4), device=DEV).tolist()


# ---------------------------------------------------------------------------------------------------------
# the engine's side
# ---------------------------------------------------------------------------------------------------------
def _part_spec(case):
    from lite_lang_b200.config.spec import PartSpec
    d, kind = _dims(case), case["kind"]
    w, h, kv = d["width"], d["heads"], d["kv"]
    if kind == "experts":
        p = dict(hidden_size=w, experts=d["experts"], top=d["top"], expert_ff=d["ff"], shared_ff=d["ff"])
        if case["design"] == "gated":
            p.update(gated=True, limit=LIMIT, shared_limit=LIMIT, swish_alpha=ALPHA, score="softmax_top",
                     router_bias=True, shared_gate=True)
        else:
            p.update(activation="relu2", score="softmax")
        return "feed_forward", PartSpec("routed_experts", p)
    if kind == "delta":
        p = dict(hidden_size=w, heads=h, kv_heads=kv, key_dim=HEAD, value_dim=HEAD, conv_taps=4, eps=1e-6)
        if case["design"] == "channel":
            p.update(decay="channel", gate="sigmoid", decay_rank=64, gate_rank=64)
        return "mixer", PartSpec("gated_delta_rule", p)
    if kind == "linear":
        p = dict(hidden_size=w, heads=h, key_dim=HEAD, value_dim=HEAD, decay=_decays(h), eps=1e-6)
        if case["design"] == "linear":
            return "mixer", PartSpec("decay_linear_attention", p)
        p.update(key_scale=HEAD ** -0.5, position=PartSpec("rope_computed", dict(
            rotary_dim=HEAD, theta=1e6, layout="half_split")))
        return "mixer", PartSpec("retention", p)
    if kind == "latent":
        rot = _rot(case)
        p = dict(hidden_size=w, heads=h, dim=HEAD - rot, rot_dim=rot, vdim=HEAD, kv_rank=d["rank"],
                 scale=HEAD ** -0.5, eps=1e-6)
        if case["design"] == "window":
            p.update(window=d["window"], rot_base=1e6, rot_dims=rot)
        else:
            p.update(window=None, q_rank=d["q_rank"])
        return "mixer", PartSpec("latent_attention", p)
    return "mixer", PartSpec("modulated_attention", dict(
        hidden_size=w, num_heads=h, num_kv_heads=kv, head_dim=HEAD, scale=HEAD ** -0.5, mask="window",
        mask_size=d["window"], keep_first=KEEP_FIRST, channel_gate=True, sink="learned",
        distance_bias=dict(max=4.0 * d["window"], buckets=BIAS_ROWS)))


def _fill_pages(storage, manager, slots, contexts, cached):
    """The requests' cached rows into the pages they hold."""
    keys, values = cached
    for src, pool in ((keys, storage.k[0]), (values, storage.v.get(0))):
        if src is None:
            continue
        for i, (slot, n) in enumerate(zip(slots, contexts)):
            pages = torch.tensor(manager.pages_of(0, slot)[:(n + PAGE - 1) // PAGE], device=DEV)
            live = pages >= 0                                  # (pages that a window has passed were given back)
            rows = torch.zeros((src.shape[0], pages.numel() * PAGE) + tuple(src.shape[3:]), dtype=pool.dtype, device=DEV)
            rows[:, :n] = src[:, i, :n]
            rows = rows.view(src.shape[0], pages.numel(), PAGE, src.shape[3], src.shape[4]).permute(0, 1, 3, 2, 4)
            pool[:, pages[live]] = rows[:, live].contiguous()


def prepare(case, seed):
    torch.cuda.set_device(0)
    return _prepare_model(case, seed) if case["kind"] == "qwen2" else _prepare_part(case, seed)


def _prepare_model(case, seed):
    from lite_lang_b200.cache.manager import CacheManager
    from lite_lang_b200.config import config_from_dict
    from lite_lang_b200.engine.model import CausalLM
    from lite_lang_b200.engine.runner import ModelRunner
    d = _dims(case)
    cfg = config_from_dict(dict(
        architectures=["Qwen2ForCausalLM"], hidden_size=d["width"], num_hidden_layers=case["layers"],
        num_attention_heads=d["heads"], num_key_value_heads=d["kv"], intermediate_size=d["inter"],
        vocab_size=d["vocab"], rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=True,
        max_position_embeddings=32768, use_sliding_window=False, torch_dtype="bfloat16"))
    model = CausalLM(cfg.model_spec())
    weights = _weights(case, seed)
    model.load(weights.pop, getattr(torch, case["dtype"]), torch.device(DEV, 0))
    decode = case["mode"] == "decode"
    batch, most = case["batch"], 8192 if decode else case["tokens"]
    per_request = (most + PAGE - 1) // PAGE
    manager = CacheManager(model.cache_groups, [batch * per_request + batch], PAGE, batch, most)
    runner = ModelRunner(model, manager, torch.device(DEV, 0), 2048, True)
    state = dict(kind="decode" if decode else "prefill", runner=runner, manager=manager, case=case,
                 tokens=_tokens(case, seed))
    if decode:
        state["contexts"] = _contexts(case)
        _open_requests(state)
        run(state)                                  # the step's graph is captured once, before a server takes requests
        for s in reversed(state["slots"]):
            manager.close(s)
        _open_requests(state)
        _fill_pages(runner.storage, manager, state["slots"], state["contexts"], _cached(case, seed))
    else:
        at, state["prompts"] = 0, []
        for n in _lengths(case):
            state["prompts"].append(state["tokens"][at:at + n])
            at += n
    return state


def _open_requests(state):
    """Requests that hold their contexts and have room up to the longest one there may be."""
    manager = state["manager"]
    state["slots"] = [manager.open() for _ in state["contexts"]]
    for s, c in zip(state["slots"], state["contexts"]):
        manager.reserve(s, manager.max_model_len)
        manager.advance(s, c)


def _prepare_part(case, seed):
    from lite_lang_b200 import ops
    from lite_lang_b200.cache.manager import CacheManager, PagedGroupSpec, StateGroupSpec
    from lite_lang_b200.cache.storage import CacheStorage
    from lite_lang_b200.csrc.build import load_library
    from lite_lang_b200.engine.batch import BatchBuilder, StepEntry
    from lite_lang_b200.parts.base import PagedKVNeed, build_part
    import lite_lang_b200.parts  # noqa: F401  (registers the parts)
    device = torch.device(DEV, 0)
    ops.configure_matmul_precision()
    family, spec = _part_spec(case)
    part = build_part(family, spec)
    weights = _weights(case, seed)
    part.load(weights.pop, torch.bfloat16, device)
    if family == "mixer":
        part.prepare(device, torch.bfloat16)
    for lib in part.kernel_libraries():
        load_library(lib)
    decode = case["mode"] == "decode"
    contexts = _contexts(dict(case, context=case.get("context", 1))) if decode else [0] * len(_lengths(case))
    new = [1] * len(contexts) if decode else _lengths(case)
    longest = max(c + n for c, n in zip(contexts, new))
    need = part.cache_need() if family == "mixer" else None
    groups, pages = [], []
    if isinstance(need, PagedKVNeed):
        groups = [PagedGroupSpec(need.num_kv_heads, need.head_dim, need.window, 1,
                                 need.head_dim if need.value_head_dim is None else need.value_head_dim, need.chunk,
                                 need.keep_first)]
        pages = [sum((c + n + PAGE - 1) // PAGE for c, n in zip(contexts, new)) + 1]
    elif need is not None:
        groups = [StateGroupSpec(tuple(need.shape), need.dtype, 1)]
    manager = CacheManager(groups, pages, PAGE, len(contexts), longest)
    storage = CacheStorage(manager, torch.bfloat16, device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    builder = BatchBuilder(manager, max(sum(new), len(new)), len(new), device, status)
    slots = [manager.open() for _ in new]
    for s, c, n in zip(slots, contexts, new):
        manager.reserve(s, c + n)
        manager.advance(s, c)
    storage.sync()
    batch = builder.build([StepEntry(s, [0] * n) for s, n in zip(slots, new)], pad_entries=len(new) if decode else None)
    cache, record = None, None
    if pages:
        if decode:
            _fill_pages(storage, manager, slots, contexts, _cached(case, seed))
        cache = storage.paged_view(0, 0, batch.slot_maps[0], True)
        record = cache.k
    elif need is not None:
        cache = storage.state_view(0, 0, True)
        record = cache.state
    first = None
    if decode and record is not None and not pages:
        matrix, taps = _cached(case, seed)
        first = matrix.reshape(len(slots), -1)
        if taps is not None:
            first = torch.cat([first, taps.reshape(len(slots), -1)], dim=1)
        record[slots] = first
        first = record.clone()
    x = _rows(case, seed)
    state = dict(kind="part", part=part, x=x, batch=batch, cache=cache, record=record, status=status,
                 manager=manager, storage=storage, builder=builder, fresh=not decode and need is not None and not pages,
                 graph=None)
    if decode:
        batch.captured = True
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                _forward(state)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = _forward(state)
        state["graph"] = graph
        if first is not None:
            record.copy_(first)
    return state


def _forward(state):
    """One call of the part, as a block makes it; what it hands on as one tensor."""
    from lite_lang_b200.parts.base import whole_output
    part, x = state["part"], state["x"]
    if state["cache"] is None:
        out = part.forward(x, state["batch"])
    else:
        out = part.forward(x, state["batch"], state["cache"])
    return whole_output(out, x.dtype)


def run(state):
    if state["kind"] == "part":
        if state["graph"] is not None:
            state["graph"].replay()
            out = state["out"]
        else:
            if state["fresh"]:
                state["record"].zero_()            # new requests: their records start at zero
            out = _forward(state)
        return {"out": out} if state["record"] is None else {"out": out, "cache": state["record"]}
    from lite_lang_b200.engine.batch import StepEntry
    runner, manager = state["runner"], state["manager"]
    if state["kind"] == "decode":
        if manager.length(state["slots"][0]) + 1 > manager.max_model_len:       # the requests have reached their limit
            for s in reversed(state["slots"]):
                manager.close(s)
            _open_requests(state)
        return {"logits": runner.step([StepEntry(s, [t], (0,)) for s, t in zip(state["slots"], state["tokens"])])}
    slots = [manager.open() for _ in state["prompts"]]
    for s, p in zip(slots, state["prompts"]):
        runner.reserve(s, len(p))
    logits = runner.step([StepEntry(s, p, (len(p) - 1,)) for s, p in zip(slots, state["prompts"])])
    for s in reversed(slots):
        manager.close(s)
    return {"logits": logits, "keys": runner.storage.k[0], "values": runner.storage.v[0]}


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------
def work(case):
    d, kind, decode = _dims(case), case["kind"], case["mode"] == "decode"
    w, h, kv = d["width"], d["heads"], d["kv"]
    n = case["batch"] if decode else case["tokens"]
    size = 4 if case.get("dtype") == "float32" else 2
    if decode:
        pairs = sum(c + 1 for c in _contexts(dict(case, context=case.get("context", 1))))
        cached = pairs
    else:
        pairs = sum(t * (t + 1) // 2 for t in _lengths(case))
        cached = n
    if kind == "qwen2":
        layer = w * (2 * h + 2 * kv) * HEAD + 3 * w * d["inter"]
        rows = case["batch"]
        flops = case["layers"] * (2 * n * layer + 4 * pairs * h * HEAD) + 2 * rows * w * d["vocab"]
        nbytes = size * (case["layers"] * (layer + 2 * cached * kv * HEAD) + w * d["vocab"]) + 4 * rows * d["vocab"]
        return {"bytes": nbytes, "flops": flops}
    if kind == "experts":
        mats = 3 if case["design"] == "gated" else 2
        one = mats * d["ff"] * w
        used = min(d["experts"], n * d["top"])
        return {"bytes": 2 * ((used + 1) * one + 2 * n * w), "flops": 2 * n * (d["top"] + 1) * one}
    window = d["window"]
    if kind in ("delta", "linear"):
        if kind == "delta":
            proj = (2 * kv + 2 * h) * HEAD if case["design"] == "head" else (2 * kv + h) * HEAD + 128
            weights = w * proj + w * h * HEAD + (0 if case["design"] == "head" else 2 * 64 * h * HEAD)
            per_state = 8
        else:
            weights, per_state = w * 5 * h * HEAD, 5
        records = len(_lengths(case)) if not decode else n
        return {"bytes": 2 * (weights + 2 * n * w) + 4 * records * h * HEAD * HEAD * (2 if decode else 1),
                "flops": 2 * n * weights + n * h * HEAD * HEAD * per_state}
    if kind == "latent":
        weights = w * h * HEAD * 2 + w * (d["rank"] + _rot(case)) + 2 * h * HEAD * d["rank"]
        if case["design"] == "full":
            weights += d["q_rank"] * (w + h * HEAD) - w * h * HEAD
        if case["design"] == "window":
            pairs, cached = _windowed(case, window, 0)
        width = d["rank"] + _rot(case)
        return {"bytes": 2 * (weights + cached * width + 2 * n * w),
                "flops": 2 * n * weights + 2 * pairs * h * (HEAD + HEAD)}
    weights = w * (3 * h + 2 * kv) * HEAD
    pairs, cached = _windowed(case, window, KEEP_FIRST)
    return {"bytes": 2 * (weights + 2 * cached * kv * HEAD + 2 * n * w), "flops": 2 * n * weights + 4 * pairs * h * HEAD}


def _windowed(case, window, keep):
    """(pairs of a query and a key it sees, cached rows that are read) with a window and kept first tokens."""
    if case["mode"] == "decode":
        seen = [min(c + 1, window) + min(keep, max(0, c + 1 - window)) for c in _contexts(case)]
        return sum(seen), sum(seen)
    pairs = 0
    for t in _lengths(case):
        for p in range(t):
            pairs += min(p + 1, window) + min(keep, max(0, p + 1 - window))
    return pairs, case["tokens"]


def tolerance(case):
    """What another correct order of the sums may differ by: about four times the error against 64 bits (``exact``)
    that was measured, which is what rounding to the storage type costs along the way."""
    if case["kind"] == "qwen2":
        if case["dtype"] == "float32":
            return {"rel": 2e-5, "max": 2e-4}       # measured 2e-6 to 5e-6
        # measured 0.010 (4 layers) and 0.015 (28, one behind the other); the same prompt twice differs by 0.013,
        # since the attention's parts of a long prompt are added up in the order in which they finish
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.016, "max": 0.5}               # measured 0.003 to 0.0045, and 0.002 in the state records


# ---------------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------------------
def exact(case, seed):
    """What ``run`` returns on a new state, in float64 (the caches' layout is the engine's own: None in their place)."""
    f = {"qwen2": _exact_qwen2, "experts": _exact_experts, "delta": _exact_delta, "linear": _exact_linear,
         "latent": _exact_latent, "shaped": _exact_shaped}[case["kind"]]
    with torch.no_grad():
        out = f(case, seed)
    if case["kind"] == "qwen2":
        return {"logits": out} if case["mode"] == "decode" else {"logits": out, "keys": None, "values": None}
    if case["kind"] == "experts":
        return {"out": out}
    if isinstance(out, tuple):
        return {"out": out[0], "cache": out[1]}
    return {"out": out, "cache": None}


def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(dims, theta, positions):
    """The model's own angles: a float32 position times a float32 frequency, rounded to float32."""
    freq = (1.0 / theta ** (torch.arange(0, dims, 2, dtype=torch.float64, device=DEV) / dims)).float()
    return (positions.float()[:, None] * freq[None, :]).double()


def _turn_halves(x, positions, theta=1e6):
    a = _angles(x.shape[-1], theta, positions)
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    lo, hi = x.chunk(2, dim=-1)
    return torch.cat((lo * c - hi * s, lo * s + hi * c), dim=-1)


def _turn_pairs(x, positions, theta=1e6):
    a = _angles(x.shape[-1], theta, positions)
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    even, odd = x[..., 0::2], x[..., 1::2]
    return torch.stack((even * c - odd * s, even * s + odd * c), dim=-1).flatten(-2)


def _spans(case):
    """(first row, rows, cached tokens before them) of each request's part of the step."""
    if case["mode"] == "decode":
        return [(i, 1, c) for i, c in enumerate(_contexts(dict(case, context=case.get("context", 1))))]
    at, out = 0, []
    for n in _lengths(case):
        out.append((at, n, 0))
        at += n
    return out


def _positions(case):
    return torch.cat([torch.arange(c, c + n, device=DEV) for _, n, c in _spans(case)])


def _seen(n, ctx, window=None, keep=0):
    q = torch.arange(ctx, ctx + n, device=DEV)[:, None]
    k = torch.arange(ctx + n, device=DEV)[None, :]
    ok = k <= q
    if window is not None:
        ok = ok & ((q - k < window) | (k < keep))
    return ok, q - k


def _heads_attention(q, k, v, scale, ok, bias=None, sink=None):
    """q [n, h, d], k and v [m, kv, d] -> [n, h, d of v]; a head at a time."""
    group = q.shape[1] // k.shape[1]
    out = []
    for a in range(q.shape[1]):
        s = (q[:, a] @ k[:, a // group].t()) * scale
        if bias is not None:
            s = s + bias[a]
        s = s.masked_fill(~ok, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[a].expand(s.shape[0], 1)), dim=1)
        p = torch.softmax(s, dim=-1)
        out.append(p[:, :k.shape[0]] @ v[:, a // group])
    return torch.stack(out, dim=1)


def _exact_qwen2(case, seed):
    d, W = _dims(case), _weights(case, seed)
    h, kv = d["heads"], d["kv"]
    table = W["model.embed_tokens.weight"]
    x = table[torch.tensor(_tokens(case, seed), device=DEV)].double()
    pos, spans = _positions(case), _spans(case)
    cached = _cached(case, seed) if case["mode"] == "decode" else None
    for i in range(case["layers"]):
        w = {n[len(f"model.layers.{i}."):]: t.double() for n, t in W.items() if n.startswith(f"model.layers.{i}.")}
        y = _rms(x) * w["input_layernorm.weight"]
        q, k, v = (y @ w[f"self_attn.{c}_proj.weight"].t() + w[f"self_attn.{c}_proj.bias"] for c in "qkv")
        q = _turn_halves(q.view(-1, h, HEAD), pos)
        k = _turn_halves(k.view(-1, kv, HEAD), pos)
        v = v.view(-1, kv, HEAD)
        att = []
        for r, (at, n, ctx) in enumerate(spans):
            kk, vv = k[at:at + n], v[at:at + n]
            if ctx:
                kk = torch.cat((cached[0][i, r, :ctx].double(), kk))
                vv = torch.cat((cached[1][i, r, :ctx].double(), vv))
            att.append(_heads_attention(q[at:at + n], kk, vv, HEAD ** -0.5, _seen(n, ctx)[0]))
        x = x + torch.cat(att).flatten(1) @ w["self_attn.o_proj.weight"].t()
        y = _rms(x) * w["post_attention_layernorm.weight"]
        gate, up = y @ w["mlp.gate_proj.weight"].t(), y @ w["mlp.up_proj.weight"].t()
        x = x + (gate * torch.sigmoid(gate) * up) @ w["mlp.down_proj.weight"].t()
    last = torch.tensor([at + n - 1 for at, n, _ in spans], device=DEV)
    y = _rms(x[last]) * W["model.norm.weight"].double()
    return torch.cat([y @ part.double().t() for part in table.split(16384)], dim=1)


def _exact_experts(case, seed):
    d, W = _dims(case), _weights(case, seed)
    x = _rows(case, seed).double()
    gated = case["design"] == "gated"

    def expert(name, rows):
        up = rows @ W[name + ".up"].double().t()
        if gated:
            a = (rows @ W[name + ".gate"].double().t()).clamp(max=LIMIT)
            hidden = a * torch.sigmoid(ALPHA * a) * (up.clamp(-LIMIT, LIMIT) + 1)
        else:
            hidden = up.clamp(min=0) ** 2
        return hidden @ W[name + ".down"].double().t()

    logits = x @ W["router"].double().t()
    if gated:
        logits = logits + W["router.b"].double()
        top, idx = logits.topk(d["top"], dim=1)
        weight = torch.softmax(top, dim=1)
    else:
        weight, idx = torch.softmax(logits, dim=1).topk(d["top"], dim=1)
    out = expert("shared", x)
    if gated:
        out = out * torch.sigmoid(x @ W["shared.sg"].double().t())
    for e in range(d["experts"]):
        rows, place = (idx == e).nonzero(as_tuple=True)
        if rows.numel():
            out[rows] += weight[rows, place][:, None] * expert(f"e{e}", x[rows])
    return out


def _exact_delta(case, seed):
    d, W = _dims(case), {n: t.double() for n, t in _weights(case, seed).items()}
    h, kv = d["heads"], d["kv"]
    x, spans = _rows(case, seed).double(), _spans(case)
    decode, channel = case["mode"] == "decode", case["design"] == "channel"
    matrix, taps = (t.double() for t in _cached(case, seed)) if decode else (None, None)
    raw = torch.cat([x @ W[n].t() for n in "qkv"], dim=1)
    filt = torch.cat([W[n + ".conv"] for n in "qkv"])                  # [channels, 4], the last tap the token's own
    a = x @ W["a1"].t() @ W["a2"].t() if channel else x @ W["a"].t()
    gate = x @ W["g1"].t() @ W["g2"].t() if channel else x @ W["g"].t()
    rate = torch.exp(W["A_log"])
    if channel:
        rate = rate.repeat_interleave(HEAD)
    decay = torch.exp(-rate * torch.nn.functional.softplus(a + W["dt_bias"]))
    decay = decay.view(-1, h, HEAD) if channel else decay[:, :, None]
    beta = torch.sigmoid(x @ W["b"].t())
    # (requests go side by side, each until its own end)
    longest = max(n for _, n, _ in spans)
    q, k, v = [], [], []
    last = []
    for r, (at, n, _) in enumerate(spans):
        before = taps[r] if decode else torch.zeros((3, raw.shape[1]), dtype=torch.float64, device=DEV)
        rows = torch.cat((before, raw[at:at + n]))
        y = sum(rows[j:j + n] * filt[:, j] for j in range(4))
        y = y * torch.sigmoid(y)
        qq, kk, vv = y.split([kv * HEAD, kv * HEAD, h * HEAD], dim=1)
        unit = [t.view(n, kv, HEAD) / torch.sqrt((t.view(n, kv, HEAD) ** 2).sum(-1, keepdim=True) + 1e-6)
                for t in (qq, kk)]
        q.append(unit[0].repeat_interleave(h // kv, dim=1) * HEAD ** -0.5)
        k.append(unit[1].repeat_interleave(h // kv, dim=1))
        v.append(vv.view(n, h, HEAD))
        last.append(rows[n:])
    S = matrix.clone() if decode else torch.zeros((len(spans), h, HEAD, HEAD), dtype=torch.float64, device=DEV)
    o = torch.zeros((x.shape[0], h, HEAD), dtype=torch.float64, device=DEV)
    order = sorted(range(len(spans)), key=lambda r: -spans[r][1])
    for t in range(longest):
        live = [r for r in order if spans[r][1] > t]
        rows = torch.tensor([spans[r][0] + t for r in live], device=DEV)
        kt, qt = torch.stack([k[r][t] for r in live]), torch.stack([q[r][t] for r in live])
        vt = torch.stack([v[r][t] for r in live])
        s = S[live] * decay[rows][:, :, None, :]                      # [request, head, value column, key channel]
        u = beta[rows][:, :, None] * (vt - (s @ kt[..., None])[..., 0])
        s = s + u[..., None] * kt[:, :, None, :]
        S[live] = s
        o[rows] = (s @ qt[..., None])[..., 0]
    act = torch.sigmoid(gate) if channel else gate * torch.sigmoid(gate)
    out = ((_rms(o) * W["norm"]).flatten(1) * act) @ W["o"].t()
    record = torch.cat((S.reshape(len(spans), -1), torch.stack(last).reshape(len(spans), -1)), dim=1)
    return out, record


def _exact_linear(case, seed):
    d, W = _dims(case), {n: t.double() for n, t in _weights(case, seed).items()}
    h, x, spans = d["heads"], _rows(case, seed).double(), _spans(case)
    keep = case["design"] == "retention"
    q, k, v, gate = (x @ W[n].t() for n in "qkvg")
    if not keep:
        q, k, v = (t * torch.sigmoid(t) for t in (q, k, v))
    q, k, v = (t.view(-1, h, HEAD) for t in (q, k, v))
    if keep:
        pos = _positions(case)
        q, k = _turn_halves(q, pos), _turn_halves(k, pos) * HEAD ** -0.5
    decay = torch.tensor(_decays(h), dtype=torch.float32, device=DEV).double()
    matrix = _cached(case, seed)[0].double() if case["mode"] == "decode" else None
    o, last = torch.zeros_like(v), []
    for r, (at, n, _) in enumerate(spans):
        i = torch.arange(n, device=DEV, dtype=torch.float64)
        S = matrix[r] if matrix is not None else torch.zeros((h, HEAD, HEAD), dtype=torch.float64, device=DEV)
        end = []
        for a in range(h):
            gap = i[:, None] - i[None, :]
            score = (q[at:at + n, a] @ k[at:at + n, a].t()) * torch.where(gap >= 0, decay[a] ** gap.clamp(min=0), 0.0)
            o[at:at + n, a] = score @ v[at:at + n, a] + decay[a] ** (i + 1)[:, None] * (q[at:at + n, a] @ S[a].t())
            end.append(decay[a] ** n * S[a] + (v[at:at + n, a] * decay[a] ** (n - 1 - i)[:, None]).t() @ k[at:at + n, a])
        last.append(torch.stack(end))
    if keep:
        y = _rms(o).flatten(1) * gate * torch.sigmoid(gate)
    else:
        y = _rms(o.flatten(1)) * W["norm"] * torch.sigmoid(gate)
    return y @ W["o"].t(), torch.stack(last).reshape(len(spans), -1)


def _exact_latent(case, seed):
    d, W = _dims(case), {n: t.double() for n, t in _weights(case, seed).items()}
    h, rot, R = d["heads"], _rot(case), d["rank"]
    x, spans, pos = _rows(case, seed).double(), _spans(case), _positions(case)
    q = x @ W["q"].t() if "q" in W else (_rms(x @ W["dq"].t()) * W["dq.norm"]) @ W["uq"].t()
    q = q.view(-1, h, HEAD)
    row = x @ W["dkv"].t()
    c, part = _rms(row[:, :R]) * W["dkv.norm"], row[:, R:]
    if rot:
        q = torch.cat((q[..., :HEAD - rot], _turn_pairs(q[..., HEAD - rot:], pos)), dim=-1)
        part = _turn_pairs(part[:, None, :], pos)[:, 0]
    cached = _cached(case, seed)[0][0, :, :, 0].double() if case["mode"] == "decode" else None
    out = []
    for r, (at, n, ctx) in enumerate(spans):
        cc, pp = c[at:at + n], part[at:at + n]
        if ctx:
            cc = torch.cat((cached[r, :ctx, :R], cc))
            pp = torch.cat((cached[r, :ctx, R:], pp))
        k = (cc @ W["uk"].t()).view(-1, h, HEAD - rot)
        if rot:
            k = torch.cat((k, pp[:, None, :].expand(-1, h, -1)), dim=-1)
        v = (cc @ W["uv"].t()).view(-1, h, HEAD)
        ok = _seen(n, ctx, d["window"] if case["design"] == "window" else None)[0]
        out.append(_heads_attention(q[at:at + n], k, v, HEAD ** -0.5, ok))
    return torch.cat(out).flatten(1) @ W["o"].t()


def _exact_shaped(case, seed):
    d, W = _dims(case), {n: t.double() for n, t in _weights(case, seed).items()}
    h, kv, window = d["heads"], d["kv"], d["window"]
    x, spans = _rows(case, seed).double(), _spans(case)
    q, k, v = (x @ W[n].t() for n in "qkv")
    q, k, v = q.view(-1, h, HEAD), k.view(-1, kv, HEAD), v.view(-1, kv, HEAD)
    cached = _cached(case, seed) if case["mode"] == "decode" else None
    half, far = BIAS_ROWS // 2, 4.0 * window
    longest = max(n + c for _, n, c in spans)
    bucket = [n if n < half else min(BIAS_ROWS - 1, half + int(math.floor(
        math.log(n / half) / math.log(far / half) * (BIAS_ROWS - half)))) for n in range(longest)]
    by_distance = W["rel"][torch.tensor(bucket, device=DEV)]                 # [distance, head]
    out = []
    for r, (at, n, ctx) in enumerate(spans):
        kk, vv = k[at:at + n], v[at:at + n]
        if ctx:
            kk = torch.cat((cached[0][0, r, :ctx].double(), kk))
            vv = torch.cat((cached[1][0, r, :ctx].double(), vv))
        ok, gap = _seen(n, ctx, window, KEEP_FIRST)
        bias = by_distance[gap.clamp(min=0)].permute(2, 0, 1)
        out.append(_heads_attention(q[at:at + n], kk, vv, HEAD ** -0.5, ok, bias, W["sink"]))
    return (torch.cat(out).flatten(1) * torch.sigmoid(x @ W["g"].t())) @ W["o"].t()
