"""The work whose time this framework is judged by: the calls that a serving program makes of it.

Two cases are whole models through `Engine.step`; the others are single mixers and feed-forwards of
the designs that the engine serves, built from their specs and run over a packed step, each with a
tolerance of its own.  The sizes are those of `crucible_b200/config/presets.py`: the 120M shape, and
the comparison shapes of width 1,024 (8 heads, 2 key/value heads) and 2,048 (16 and 4), with heads of
128 or 64.  `listed()` says what each case stands for; `draw` takes other sizes of the same ranges.

A case's step: `new` tokens of the longest prompt portion, brought by `requests` requests (their
lengths fall unevenly if there are several); `decoding` requests more that bring one token each
behind `held` cached tokens (uneven as well); then `more` steps in which every request brings one
token.  Steps in which every request brings one token are captured once and replayed, as the engine
does with them; portions run as they come.  A pass begins with what the engine does when it hands
out a request slot: the state is zeroed.
"""
from __future__ import annotations

import json
import math
import os
import tempfile

import torch

DEV = "cuda:0"
PAGE = 16
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
RECURRENT = ("gated_delta", "channel_delta", "mlstm", "wkv", "mamba2", "retention")
ATTENTION = ("attention", "sink_attention", "latent_attention")
EPS, TAPS, VOCAB, EXPERTS, TOP = 1e-5, 4, 50304, 8, 2
ROT, RANK, LOW = 64, 192, 64           # latent rows: 192 of latent, 64 rotated; the low ranks


def _case(name, part, **given):
    case = {"name": name, "part": part, "dtype": "bfloat16", "width": 2048, "heads": 16, "kv_heads": 4, "dim": 128,
            "requests": 1, "new": 0, "decoding": 0, "held": 0, "more": 0, "window": 0, "sink": False,
            "scattered": False}
    case.update(given)
    if name is None:
        del case["name"]
    return case


def listed():
    return [
        # a document read by the 120M shape: the engine's whole prompt step (12 layers and the head)
        _case("dense-prefill", "model", new=2048),
        # short turns of eight users of the 120M shape: uneven prompts, then eight tokens for each
        _case("dense-chat", "model", requests=8, new=180, more=8),
        # the 32-bit engine, with which results are checked: a middling odd portion, one layer's attention
        _case("float32-portion", "attention", dtype="float32", width=768, heads=12, kv_heads=4, dim=64, new=700),
        # latent attention, a long prompt; and the smallest call: one user's next token
        _case("latent-prefill", "latent_attention", new=2048, sink=True),
        _case("latent-decode-1", "latent_attention", width=1024, heads=8, decoding=1, held=3001, scattered=True),
        # windowed grouped attention with a gate: a long prompt; and a server's mixed step,
        # a ragged portion beside users who are decoding
        _case("window-prefill", "sink_attention", new=2048, window=1024),
        _case("window-mixed", "sink_attention", new=509, decoding=24, held=2000, window=1024, scattered=True),
        # mixers with a matrix memory: a long prompt through the delta rule, three uneven prompts
        # through the mLSTM, and the short prompts and next tokens of 32 users of the state-space rule
        _case("delta-prefill", "gated_delta", new=2048),
        _case("mlstm-portions", "mlstm", width=1024, heads=8, requests=3, new=1337),
        _case("state-space-decode-32", "mamba2", kv_heads=2, requests=32, new=24, more=4),
        # routed experts with a shared one: a long prompt's rows, and eight users' next tokens
        _case("experts-prefill", "experts", new=2048),
        _case("experts-decode-8", "experts", decoding=8, held=1),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    part = rng.choice(("model", "attention", "sink_attention", "sink_attention", "latent_attention", "latent_attention",
                       "experts", "experts") + RECURRENT)
    wide = rng.random() < 0.5
    given = dict(width=2048, heads=16, kv_heads=4) if wide else dict(width=1024, heads=8, kv_heads=2)
    given["dim"] = rng.choice((64, 128, 128))
    given["scattered"] = rng.random() < 0.5
    if part == "model":
        if rng.random() < 0.5:
            return _case(None, part, new=_spread(rng, 16, 2048))
        return _case(None, part, requests=rng.randint(1, 8), new=_spread(rng, 8, 200), more=rng.randint(1, 8))
    if part == "mamba2":
        given["kv_heads"] = rng.choice((1, 2))
    if part == "experts":
        return _case(None, part, new=_spread(rng, 1, 2048), **given)
    if rng.random() < 0.15:
        given.update(dtype="float32", width=1024, heads=8, kv_heads=min(2, given["kv_heads"]))
    longest = 2048 if given.get("dtype") is None else 700
    if part in RECURRENT:
        most = 64 // given["heads"] if part == "mlstm" else 48
        if rng.random() < 0.6:
            return _case(None, part, requests=min(most, rng.choice((1, 1, 2, 5))), new=_spread(rng, 17, longest), **given)
        return _case(None, part, requests=_spread(rng, 1, most), new=rng.randint(1, 30), more=rng.randint(2, 5), **given)
    if part == "sink_attention":
        given["window"] = rng.choice((0, 512, 1024))
    if part == "latent_attention":
        given.update(window=rng.choice((0, 0, 1024)), sink=rng.random() < 0.5)
    kind = rng.random()
    if kind < 0.45:
        return _case(None, part, requests=rng.choice((1, 1, 3)), new=_spread(rng, 40, longest), **given)
    if kind < 0.8:
        return _case(None, part, decoding=_spread(rng, 1, 48), held=_spread(rng, 100, 3800), **given)
    return _case(None, part, new=_spread(rng, 40, longest), decoding=rng.randint(1, 24), held=_spread(rng, 100, 3000),
                 **given)


# ---------------------------------------------------------------------------
# the steps of a case
# ---------------------------------------------------------------------------

def _uneven(longest, i):
    return longest - (i * 577) % longest


def _requests(case):
    """(tokens held before the pass, tokens of the first step) for every request, decoding ones first."""
    out = [(_uneven(case["held"], i), 1) for i in range(case["decoding"])]
    if case["new"]:
        out += [(0, _uneven(case["new"], i)) for i in range(case["requests"])]
    return out


def _schedule(case):
    first = _requests(case)
    return [[n for _, n in first]] + [[1] * len(first)] * case["more"]


def _rows(case):
    return sum(sum(step) for step in _schedule(case))


def _generator(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + salt)


# ---------------------------------------------------------------------------
# parts: specs, weights
# ---------------------------------------------------------------------------

def _build(case):
    from crucible_b200.config.model_config import FeedForwardSpec, MixerSpec, PositionSpec
    from crucible_b200.parts import FEED_FORWARDS, MIXERS
    part, W, H, G, D = case["part"], case["width"], case["heads"], case["kv_heads"], case["dim"]
    if part == "experts":
        ff = W * 11 // 8                           # half of the dense feed-forward's width
        return FEED_FORWARDS.build("moe", FeedForwardSpec("moe", W, ff, (("experts", EXPERTS), ("top", TOP),
                                                                         ("shared_intermediate", ff))))
    position, scale, window, extra = None, D ** -0.5, case["window"] or None, ()
    if part == "attention":
        position = PositionSpec("rope", D, 10000.0, 4096)
    elif part == "sink_attention":
        position = PositionSpec("rope_interleaved", D // 2, 500000.0, 0)
        extra = (("sink", 0), ("gate", "element"), ("qk_norm_eps", EPS))
    elif part == "latent_attention":
        G, scale, position = 1, (D + ROT) ** -0.5, PositionSpec("rope_interleaved", ROT, 10000.0, 0)
        extra = (("rot_dim", ROT), ("value_dim", D), ("kv_rank", RANK), ("norm_eps", EPS), ("gate", "element"),
                 ("q_rank", W // 2), ("sink", case["sink"]))
    elif part == "retention":
        position = PositionSpec("rope_halves", D, 10000.0, 0)
        extra = (("value_dim", D), ("norm_eps", EPS), ("decay", tuple(_decays(H))))
    elif part == "mlstm":
        extra = (("value_dim", D), ("gate_cap", 15.0), ("norm_eps", EPS))
    elif part == "wkv":
        extra = (("decay_rank", LOW), ("norm_eps", EPS))
    else:
        extra = (("value_dim", D), ("conv_taps", TAPS), ("norm_eps", EPS), ("rank", LOW))
    return MIXERS.build(part, MixerSpec(part, W, H, G, D, scale, window, position, extra))


def _decays(heads):
    return [1.0 - 2.0 ** (-4 - 0.75 * (i % 8)) for i in range(heads)]


_BOUND = {}


def _bound(case):
    """The case's part with its weights laid out (they are the same for every input), and the weights."""
    key = tuple(case[k] for k in ("part", "dtype", "width", "heads", "kv_heads", "dim", "window", "sink"))
    if key not in _BOUND:
        while len(_BOUND) >= 2:
            _BOUND.pop(next(iter(_BOUND)))
        part, dtype, g = _build(case), DTYPES[case["dtype"]], _generator(7)
        tensors = {}
        for d in part.tensors():
            t = torch.randn(d.shape, generator=g, device=DEV)
            if d.init is not None:
                kind, a, b = d.init
                t = a + (b - a) * torch.rand(d.shape, generator=g, device=DEV) if kind == "uniform" else a + b * t
            elif d.role == "vector":
                t = 1.0 + 0.1 * t
            else:
                t = t * d.shape[-1] ** -0.5
            tensors[d.name] = t.to(dtype) if d.role == "matrix" else t
        part.bind(tensors, dtype, torch.device(DEV))
        _BOUND[key] = part, tensors
    return _BOUND[key]


def _inputs(case, seed):
    """The rows of every step in the layer's dtype, and the pages' contents (keys, values; None for a part
    without a cache) with every request's page table."""
    g, dtype = _generator(seed, 1), DTYPES[case["dtype"]]
    steps = [torch.randn((sum(step), case["width"]), generator=g, device=DEV).to(dtype) for step in _schedule(case)]
    if case["part"] not in ATTENTION:
        return steps, None
    latent = case["part"] == "latent_attention"
    heads, dim = (1, RANK + ROT) if latent else (case["kv_heads"], case["dim"])
    lengths = [held + n + case["more"] for held, n in _requests(case)]
    per = -(-max(lengths) // PAGE)
    pages = len(lengths) * per
    table = torch.arange(pages, device=DEV)
    if case["scattered"]:
        table = torch.randperm(pages, generator=g, device=DEV)
    shape = (1, pages + 1, heads, PAGE, dim)
    contents = [torch.randn(shape, generator=g, device=DEV).to(dtype) for _ in range(1 if latent else 2)]
    return steps, (contents, table.view(len(lengths), per))


# ---------------------------------------------------------------------------
# whole models
# ---------------------------------------------------------------------------

_ENGINE = []


def _engine():
    from crucible_b200.config.presets import shape
    from crucible_b200.engine.engine import Engine, EngineOptions
    from crucible_b200.weights import write_random_model
    if not _ENGINE:
        folder = write_random_model(shape("120m"), os.path.join(tempfile.mkdtemp(), "120m"), seed=0)
        _ENGINE.append((Engine(folder, EngineOptions(dtype="bfloat16", max_requests=8)), folder))
    return _ENGINE[0]


def _tokens(case, seed):
    lengths = [n + case["more"] for _, n in _requests(case)]
    ids = torch.randint(0, VOCAB, (sum(lengths),), generator=torch.Generator().manual_seed(int(seed))).tolist()
    out, at = [], 0
    for n in lengths:
        out.append(ids[at:at + n])
        at += n
    return out


def _run_model(state):
    from crucible_b200.engine.engine import StepEntry
    engine, case, tokens = state["engine"], state["case"], state["tokens"]
    fed, logits = [0] * len(tokens), []
    for step in _schedule(case):
        entries = [StepEntry(i, tokens[i][fed[i]:fed[i] + n], [n - 1]) for i, n in enumerate(step)]
        fed = [a + n for a, n in zip(fed, step)]
        logits.append(engine.step(entries).clone())
    for i in range(len(tokens)):
        engine.finish(i)
    return logits


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def _contexts(case, part, pages, dtype):
    """The packed steps of the case as the engine packs them: one `StepContext` a step."""
    from crucible_b200.engine.context import CacheStorage, HostStep, Scratch, StepContext, StepLayout
    from crucible_b200.parts import LayerBinding
    is_mixer = case["part"] != "experts"
    nbytes = int(part.state_bytes()) if is_mixer else 0
    need = part.cache_need() if is_mixer else None
    caches, stride = [], ()
    if need is not None:
        contents, table = pages
        storage = CacheStorage(1, contents[0].shape[1], PAGE, need.kv_heads, need.head_dim, dtype, DEV,
                               values_are_keys=need.values_are_keys)
        storage.keys(0).copy_(contents[0][0])
        if not need.values_are_keys:
            storage.values(0).copy_(contents[1][0])
        caches, stride = [storage], (table.shape[1],)
    first = _requests(case)
    n_req = len(first)
    state = torch.zeros((n_req, nbytes), dtype=torch.uint8, device=DEV) if nbytes else None
    binding = LayerBinding(group=0 if caches else None, slot=0, write=True, state_offset=0, state_bytes=nbytes)
    scratch, held, out = Scratch(DEV), [h for h, _ in first], []
    for step in _schedule(case):
        layout = StepLayout(sum(step), n_req, 0, stride)
        offsets = layout.offsets()
        meta = torch.zeros(offsets["_total"][1], dtype=torch.int32)
        after = [h + n for h, n in zip(held, step)]
        starts = [0]
        for n in step:
            starts.append(starts[-1] + n)
        given = {"positions": [h + i for h, n in zip(held, step) for i in range(n)],
                 "row_request": [r for r, n in enumerate(step) for _ in range(n)], "req_row_start": starts,
                 "req_context_len": after, "req_first_pos": held, "req_state_slot": list(range(n_req))}
        if caches:
            given["table0"] = pages[1].reshape(-1).tolist()
        for name, values in given.items():
            at, n = offsets[name]
            meta[at:at + n] = torch.tensor(values, dtype=torch.int32)
        host = HostStep(list(range(n_req)), list(step), held, after, list(range(n_req)))
        out.append(StepContext(layout=layout, meta=meta.to(DEV), caches=caches, state=state, scratch=scratch, dtype=dtype,
                               host=host))
        held = after
    return out, binding, caches, state


def _forward(case, part, ctx, h, residual, binding):
    if case["part"] == "experts":
        part.forward(ctx, h, residual)
    else:
        part.forward(ctx, h, residual, binding)


def prepare(case, seed):
    if case["part"] == "model":
        return {"case": case, "engine": _engine()[0], "tokens": _tokens(case, seed)}
    part, _ = _bound(case)
    rows, pages = _inputs(case, seed)
    ctxs, binding, caches, state = _contexts(case, part, pages, DTYPES[case["dtype"]])
    out = {"case": case, "part": part, "binding": binding, "caches": caches, "state": state, "steps": []}
    for n, ctx, h in zip(_schedule(case), ctxs, rows):
        out["steps"].append({"ctx": ctx, "h": h, "x": torch.zeros((h.shape[0], case["width"]), device=DEV), "graph": None,
                             "decode": max(n) == 1})
    if any(s["decode"] for s in out["steps"]):
        kept = [c.keys(0).clone() for c in caches], [c.values(0).clone() for c in caches]
        for s in out["steps"]:                    # sizes the scratch rows before anything is captured
            _one(out, s)
        for s in out["steps"]:
            if s["decode"]:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    _one(out, s)
                s["graph"] = graph
        for c, k, v in zip(caches, *kept):
            c.keys(0).copy_(k)
            c.values(0).copy_(v)
    return out


def _one(state, s):
    s["x"].zero_()
    _forward(state["case"], state["part"], s["ctx"], s["h"], s["x"], state["binding"])


def run(state):
    if "engine" in state:
        return _run_model(state)
    if state["state"] is not None:
        state["state"].zero_()
    for s in state["steps"]:
        if s["graph"] is not None:
            s["graph"].replay()
        else:
            _one(state, s)
    out = {"rows": [s["x"] for s in state["steps"]]}
    if state["state"] is not None:
        out["state"] = state["state"].view(torch.float32)
    for c in state["caches"]:
        out["keys"] = c.keys(0)
        if not c.values_are_keys:
            out["values"] = c.values(0)
    return out


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------

def _visible(case, held, n):
    """Keys that the n rows after `held` tokens read, over all rows; and the tokens among them."""
    w = case["window"]
    pairs = sum(min(held + i + 1, w) if w else held + i + 1 for i in range(n))
    return pairs, min(held + n, w + n - 1) if w else held + n


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    T, W, H, G, D = _rows(case), case["width"], case["heads"], case["kv_heads"], case["dim"]
    steps = _schedule(case)
    if case["part"] == "model":
        layers, W, H, G, D, ff = 12, 768, 12, 4, 64, 2048
        weights = layers * (W * (H + 2 * G) * D + H * D * W + 3 * W * ff)
        wanted = sum(len(s) for s in steps)
        flops, moved, held = 2.0 * T * weights + 2.0 * wanted * VOCAB * W, 0.0, [0] * len(steps[0])
        for step in steps:
            moved += 2.0 * (weights + VOCAB * W) + 4.0 * len(step) * VOCAB
            for i, n in enumerate(step):
                pairs, seen = _visible(dict(case, window=0), held[i], n)
                flops += layers * 4.0 * pairs * H * D
                moved += layers * 2.0 * 2 * G * D * (seen + n)
                held[i] += n
        return {"bytes": moved, "flops": flops}
    _, tensors = _sizes(case)
    if case["part"] == "experts":
        one = 3 * W * (W * 11 // 8)
        used = min(EXPERTS, T * TOP)
        return {"bytes": 2.0 * (W * EXPERTS + (used + 1) * one) + T * W * (size + 4.0),
                "flops": 2.0 * T * (W * EXPERTS + (TOP + 1) * one)}
    weights = sum(math.prod(shape) for shape in tensors)
    moved, flops = size * weights * len(steps) + T * W * (size + 4.0), 2.0 * T * weights
    held = [h for h, _ in _requests(case)]
    for step in steps:
        for i, n in enumerate(step):
            if case["part"] in ATTENTION:
                pairs, seen = _visible(case, held[i], n)
                latent = case["part"] == "latent_attention"
                moved += size * (seen + n) * (RANK + ROT if latent else 2 * G * D)
                flops += 2.0 * pairs * H * (D + ROT + D if latent else 2 * D)
                held[i] += n
            else:
                moved += 2 * 4.0 * H * D * D
                flops += 4.0 * n * H * D * D
    return {"bytes": moved, "flops": flops}


def _sizes(case):
    part = _build(case)
    return part, [d.shape for d in part.tensors()]


def tolerance(case):
    """About four times what the start shows against 64 bits (the largest over seeds and sizes)."""
    if case["part"] == "model":
        return {"rel": 2.4e-2}
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    # (a first token's result is (k . q) v, normed: where the dot product is small its rounding is not)
    return {"rel": {"experts": 8e-3, "wkv": 3e-2, "retention": 4e-2}.get(case["part"], 2e-2)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, positions, dims, base, halves, rounded=True):
    """x [T, heads, n]; angles are float32 products of position and frequency (`rounded`), or tables
    whose sines and cosines are rounded."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f = base ** (-2.0 * i / dims)
    if rounded:
        a = (positions.float()[:, None] * f.float()[None]).double()
        c, s = a.cos()[:, None], a.sin()[:, None]
    else:
        a = positions.double()[:, None] * f[None]
        c, s = a.cos().float().double()[:, None], a.sin().float().double()[:, None]
    if halves:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        turned = torch.cat([u * c - v * s, v * c + u * s], -1)
    else:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, first, scale, window, sink):
    """q [T, H, D] at positions first..., k [N, G, D], v [N, G, E] -> [T, H, E]."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        i, j = first + torch.arange(T, device=q.device)[:, None], torch.arange(k.shape[0], device=q.device)[None]
        seen = j <= i
        if window:
            seen = seen & (i - j < window)
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        p = torch.softmax(s, -1)[:, :k.shape[0]]
        out.append(p @ v[:, h * G // H])
    return torch.stack(out, 1)


def _exact_attention(case, w, steps, pages):
    W, H, G, D = case["width"], case["heads"], case["kv_heads"], case["dim"]
    (contents, table), part = pages, case["part"]
    latent = part == "latent_attention"
    cached = [c[0].double() for c in contents]                       # [pages, heads, PAGE, n]
    held = [h for h, _ in _requests(case)]
    rows = []
    for step, h_all in zip(_schedule(case), steps):
        at, out = 0, []
        for r, n in enumerate(step):
            h = h_all[at:at + n].double()
            at += n
            pos = torch.arange(held[r], held[r] + n, device=DEV)
            if part == "attention":
                q = _turn((h @ w["q"].T).view(n, H, D), pos, D, 10000.0, True, rounded=False)
                k = _turn((h @ w["k"].T).view(n, G, D), pos, D, 10000.0, True, rounded=False)
                new = [k, (h @ w["v"].T).view(n, G, D)]
            elif part == "sink_attention":
                q = _rms((h @ w["q"].T).view(n, H, D), EPS) * w["q.norm"]
                k = _rms((h @ w["k"].T).view(n, G, D), EPS) * w["k.norm"]
                q, k = (_turn(t, pos, D // 2, 500000.0, False) for t in (q, k))
                new = [k, (h @ w["v"].T).view(n, G, D)]
            else:
                q = ((_rms(h @ w["dq"].T, EPS) * w["dq.norm"]) @ w["uq"].T).view(n, H, D + ROT)
                q = torch.cat([q[..., :D], _turn(q[..., D:], pos, ROT, 10000.0, False)], -1)
                both = h @ w["dkv"].T
                c = _rms(both[:, :RANK], EPS) * w["dkv.norm"]
                new = [torch.cat([c, _turn(both[:, None, RANK:], pos, ROT, 10000.0, False)[:, 0]], -1)[:, None]]
            place = table[r][pos // PAGE]
            for stored, t in zip(cached, new):
                stored[place, :, pos % PAGE] = t
            total = held[r] + n
            every = torch.arange(total, device=DEV)
            read = [stored[table[r][every // PAGE], :, every % PAGE] for stored in cached]      # [total, heads, n]
            if latent:
                c, turned = read[0][:, 0, :RANK], read[0][:, 0, RANK:]
                k = torch.cat([(c @ w["uk"].T).view(total, H, D), turned[:, None].expand(total, H, ROT)], -1)
                v = (c @ w["uv"].T).view(total, H, D)
                sink = w["sink"] if case["sink"] else None
                o = _attend(q, k, v, held[r], (D + ROT) ** -0.5, case["window"], sink)
            else:
                sink = torch.zeros(H, dtype=torch.float64, device=DEV) if part == "sink_attention" else None
                o = _attend(q, read[0], read[1], held[r], D ** -0.5, case["window"], sink)
            o = o.reshape(n, H * D)
            if part != "attention":
                o = o * torch.sigmoid(h @ w["g"].T)
            out.append(o @ w["o"].T)
            held[r] += n
        rows.append(torch.cat(out, 0))
    out = {"rows": rows, "keys": cached[0]}
    if not latent:
        out["values"] = cached[1]
    return out


def _conv(x, taps, tail):
    """x [T, C] behind the tail [taps - 1, C]: the causal convolution, and the new tail."""
    padded = torch.cat([tail, x], 0)
    out = sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(taps.shape[1]))
    return out, padded[x.shape[0]:]


def _recurrent_inputs(case, w, h, pos, rest):
    """q, k, v [T, H, .], decay [T, H, D], the update's and the output's kind of the rule, the gate and
    what the request carries beside its matrix."""
    part, T, H, G, D = case["part"], h.shape[0], case["heads"], case["kv_heads"], case["dim"]
    wide = lambda t, n: t.repeat_interleave(H // n, 1)
    gate, extra = None, {}
    if part in ("gated_delta", "channel_delta"):
        taps = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0)
        joint, rest = _conv(h @ torch.cat([w["q"], w["k"], w["v"]], 0).T, taps, rest)
        q, k, v = _silu(joint).split([G * D, G * D, H * D], 1)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        q, k, v = wide(unit(q.view(T, G, D)) * D ** -0.5, G), wide(unit(k.view(T, G, D)), G), v.view(T, H, D)
        extra["beta"] = torch.sigmoid(h @ w["b"].T)
        if part == "gated_delta":
            rate = torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"])
            decay = torch.exp(-torch.exp(w["A_log"]) * rate)[..., None].expand(T, H, D)
            gate = _silu(h @ w["g"].T)
        else:
            rate = torch.nn.functional.softplus((h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(T, H, D)
            decay = torch.exp(-torch.exp(w["A_log"])[:, None] * rate)
            gate = torch.sigmoid((h @ w["g1"].T) @ w["g2"].T)
    elif part == "mlstm":
        q, k, v = ((h @ w[n].T).view(T, H, D) for n in "qkv")
        q = q * D ** -0.5
        cap = lambda z: 15.0 * torch.tanh(z / 15.0)
        extra["in"] = cap(h @ w["i"].T + w["i.b"])
        extra["keep"] = torch.nn.functional.logsigmoid(cap(h @ w["f"].T + w["f.b"]))
        decay, gate = None, torch.sigmoid(h @ w["g"].T)
    elif part == "wkv":
        before = torch.cat([rest, h[:-1]], 0)
        mix = {s: h + (before - h) * w[f"mu.{s}"] for s in "rkvgw"}
        rest = h[-1:]
        q, k, v = ((mix[n] @ w[n].T).view(T, H, D) for n in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"])).view(T, H, D)
        gate = _silu(mix["g"] @ w["g"].T)
    elif part == "mamba2":
        z, joint, dt = (h @ w["in"].T).split([H * D, H * D + 2 * G * D, H], 1)
        joint, rest = _conv(joint, w["conv"], rest)
        v, k, q = _silu(joint + w["conv.b"]).split([H * D, G * D, G * D], 1)
        dt = torch.nn.functional.softplus(dt + w["dt_bias"])
        q, v = wide(q.view(T, G, D), G), v.view(T, H, D)
        k = wide(k.view(T, G, D), G) * dt[..., None]
        decay, gate = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None].expand(T, H, D), z
    else:
        q, k, v = ((h @ w[n].T).view(T, H, D) for n in "qkv")
        q, k = _turn(q, pos, D, 10000.0, True), _turn(k, pos, D, 10000.0, True) * D ** -0.5
        decay = torch.tensor(_decays(H), dtype=torch.float32, device=DEV).double()[None, :, None].expand(T, H, D)
        gate = _silu(h @ w["g"].T)
    return q, k, v, decay, gate, extra, rest


def _exact_recurrent(case, w, steps):
    part, H, D = case["part"], case["heads"], case["dim"]
    n_req, f64 = len(_requests(case)), torch.float64
    tail = {"gated_delta": TAPS - 1, "channel_delta": TAPS - 1, "mamba2": TAPS - 1, "wkv": 1}.get(part, 0)
    cols = {"wkv": case["width"], "mamba2": H * D + 2 * case["kv_heads"] * D}.get(part, 2 * case["kv_heads"] * D + H * D)
    S = torch.zeros((n_req, H, D, D), dtype=f64, device=DEV)
    norm, top = torch.zeros((n_req, H, D), dtype=f64, device=DEV), torch.zeros((n_req, H), dtype=f64, device=DEV)
    rest = [torch.zeros((tail, cols), dtype=f64, device=DEV) for _ in range(n_req)]
    held, rows = [0] * n_req, []
    for step, h_all in zip(_schedule(case), steps):
        at, given = 0, []
        for r, n in enumerate(step):
            pos = torch.arange(held[r], held[r] + n, device=DEV)
            *parts, rest[r] = _recurrent_inputs(case, w, h_all[at:at + n].double(), pos, rest[r])
            given.append(parts)
            at += n
            held[r] += n
        out = [torch.zeros((n, H, D), dtype=f64, device=DEV) for n in step]
        for t in range(max(step)):                 # every request's token t together
            live = [r for r, n in enumerate(step) if n > t]
            take = lambda i: torch.stack([given[r][i][t] for r in live])
            more = lambda name: torch.stack([given[r][5][name][t] for r in live])
            q, k, v, s = take(0), take(1), take(2), S[live]
            if part == "mlstm":
                m, n_ = top[live], norm[live]
                m_new = torch.maximum(more("keep") + m, more("in"))
                a, b = torch.exp(more("keep") + m - m_new), torch.exp(more("in") - m_new)
                s = a[..., None, None] * s + (b[..., None] * k)[..., None] * v[:, :, None]
                n_ = a[..., None] * n_ + b[..., None] * k
                low = torch.maximum((n_ * q).sum(-1).abs(), torch.exp(-m_new)) + 1e-6
                o = torch.einsum("rhde,rhd->rhe", s, q) / low[..., None]
                top[live], norm[live] = m_new, n_
            elif part == "wkv":
                kv = k[..., None] * v[:, :, None]
                o = torch.einsum("rhde,rhd->rhe", s + w["u"][None, :, :, None] * kv, q)
                s = take(3)[..., None] * s + kv
            else:
                s = take(3)[..., None] * s
                u = v
                if part in ("gated_delta", "channel_delta"):
                    u = more("beta")[..., None] * (v - torch.einsum("rhde,rhd->rhe", s, k))
                s = s + k[..., None] * u[:, :, None]
                o = torch.einsum("rhde,rhd->rhe", s, q)
                if part == "mamba2":
                    o = o + w["D"][None, :, None] * v
            S[live] = s
            for i, r in enumerate(live):
                out[r][t] = o[i]
        done = []
        for r, n in enumerate(step):
            o, gate = out[r], given[r][4]
            if part == "mamba2":
                y = _rms(o.reshape(n, H * D) * _silu(gate), EPS) * w["norm"]
            else:
                y = _rms(o, EPS)
                if part in ("gated_delta", "channel_delta"):
                    y = y * w["norm"]
                y = y.reshape(n, H * D)
                if part in ("mlstm", "wkv"):
                    y = y * w["norm"]
                y = y * gate
            done.append(y @ w["o"].T)
        rows.append(torch.cat(done, 0))
    state = [S.reshape(n_req, -1)]
    if part == "mlstm":
        pad = torch.zeros((n_req, -H % 4), dtype=f64, device=DEV)
        state += [norm.reshape(n_req, -1), top, pad]
    if tail:
        state.append(torch.stack(rest).reshape(n_req, -1))
    return {"rows": rows, "state": torch.cat(state, 1)}


def _stored(path):
    """The tensors of a safetensors file: a JSON header behind its 64-bit length, then the data."""
    with open(path, "rb") as f:
        blob = f.read()
    start = 8 + int.from_bytes(blob[:8], "little")
    kinds, out = {"BF16": torch.bfloat16, "F32": torch.float32}, {}
    for name, d in json.loads(blob[8:start]).items():
        if name != "__metadata__":
            a, b = d["data_offsets"]
            t = torch.frombuffer(bytearray(blob[start + a:start + b]), dtype=kinds[d["dtype"]])
            out[name] = t.view(d["shape"]).to(DEV).double()
    return out


def _exact_model(case, seed):
    H, G, D, eps = 12, 4, 64, 1e-5
    w = _stored(os.path.join(_engine()[1], "model.safetensors"))
    names = _engine()[0].config.tensor_names
    of = lambda local, layer=None: w[names[local].format(layer=layer) if layer is not None else names[local]]
    per_request = []
    for tokens in _tokens(case, seed):
        pos = torch.arange(len(tokens), device=DEV)
        x = of("embedding.table")[torch.tensor(tokens, device=DEV)]
        for i in range(12):
            h = _rms(x, eps) * of("layer.mixer_norm.gain", i)
            q, k, v = (h @ of(f"layer.mixer.{n}", i).T for n in "qkv")
            q = _turn(q.view(-1, H, D), pos, D, 10000.0, True, rounded=False)
            k = _turn(k.view(-1, G, D), pos, D, 10000.0, True, rounded=False)
            o = _attend(q, k, v.view(-1, G, D), 0, D ** -0.5, 0, None)
            x = x + o.reshape(-1, H * D) @ of("layer.mixer.o", i).T
            h = _rms(x, eps) * of("layer.feed_forward_norm.gain", i)
            gate, up, down = (of(f"layer.feed_forward.{n}", i) for n in ("gate", "up", "down"))
            x = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
        last = x[len(tokens) - 1 - case["more"]:]
        per_request.append((_rms(last, eps) * of("final_norm.gain")) @ of("embedding.table").T)
    return [torch.stack([r[i] for r in per_request]) for i in range(case["more"] + 1)]


def _exact_experts(case, w, rows):
    out = []
    for h in (r.double() for r in rows):
        best, idx = torch.topk(h @ w["router"].T, TOP, -1)
        weight = torch.softmax(best, -1)
        ffn = lambda x, name: (_silu(x @ w[f"{name}.gate"].T) * (x @ w[f"{name}.up"].T)) @ w[f"{name}.down"].T
        y = ffn(h, "shared")
        for e in range(EXPERTS):
            t, j = (idx == e).nonzero(as_tuple=True)
            y[t] += weight[t, j, None] * ffn(h[t], f"e{e}")
        out.append(y)
    return {"rows": out}


def exact(case, seed):
    if case["part"] == "model":
        return _exact_model(case, seed)
    _, tensors = _bound(case)
    w = {k: v.double() for k, v in tensors.items()}
    rows, pages = _inputs(case, seed)
    if case["part"] == "experts":
        return _exact_experts(case, w, rows)
    if case["part"] in RECURRENT:
        return _exact_recurrent(case, w, rows)
    return _exact_attention(case, w, rows, pages)
