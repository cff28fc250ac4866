"""The recurrences over prompts' portions in chunks of 32 tokens (`csrc/recurrent_chunks.cu`), and over a
token of each of several requests (`csrc/recurrent.cu`, the step form), against the
same recurrences token by token in float64, for every rule: portions that end inside a chunk, at its
edge and one token beyond it, a state carried in, heads and values that are no whole tiles, decays of 0
and 1, requests of one token at the head of the step.  The operands are float32, so the error is that
of float32 sums: the bound is twice what the token-by-token kernel shows on the same operands (a
chunk sums in another order, the triangular system included; up to 64 chunks showed 1.5 times), or four roundings
of float32.  The mLSTM divides by a sum that may all but cancel, in either form: four times, or eight roundings."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENGTHS = [(1, 128, 33), (1, 1, 161), (200,), (129, 31, 32), (1,), (1, 1, 1, 1, 1)]
ROUNDING = 2.0 ** -23


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _ctx(lengths, dtype):
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    lead = 0
    while lead < len(lengths) and lengths[lead] == 1:
        lead += 1
    room = {}

    def scratch(name, shape, kind):
        room[name] = torch.full(tuple(shape), float("nan"), dtype=kind, device=DEV)
        return room[name]
    slots = list(range(len(lengths)))[::-1]
    return SimpleNamespace(dtype=dtype, n_requests=len(lengths), req_row_start=_i32(starts), req_state_slot=_i32(slots),
                           scratch=scratch, host=SimpleNamespace(max_new_tokens=max(lengths), lead_single=lead)), starts, slots


def _operands(rule, k, T, H, G, D, E, g):
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, kk = (torch.randn(T, G, D, generator=g) for _ in range(2))
    v = torch.randn(T, H, E, generator=g)
    w = sc0 = sc1 = per_head = None
    decay = torch.rand(T, H, generator=g) ** 0.1
    decay[3::29] = 0.0
    decay[5::31] = 1.0
    if rule in (k.DELTA, k.CHANNEL):
        q, kk, sc1 = unit(q) * D ** -0.5, unit(kk), torch.rand(T, H, generator=g)
        sc0 = decay
    if rule == k.SSD:
        sc0, sc1, per_head = decay, torch.rand(T, H, generator=g), torch.randn(H, generator=g)
    if rule == k.MLSTM:
        q = q * D ** -0.5
        sc0 = torch.nn.functional.logsigmoid(torch.randn(T, H, generator=g) * 3.0)
        sc1 = torch.randn(T, H, generator=g) * 4.0
    if rule in (k.WKV, k.CHANNEL):
        w = torch.rand(T, H, D, generator=g) ** 0.2
        w[:, :, 0], w[:, :, 1] = 1.0, 0.0
    if rule == k.WKV:
        per_head = torch.randn(H, D, generator=g)
    return q, kk, v, w, sc0, sc1, per_head


def _walk(rule, k, q, kk, v, w, sc0, sc1, per_head, S, n, m):
    """One request's tokens in float64."""
    H, out = v.shape[1], torch.zeros(v.shape, dtype=torch.float64)
    rep = H // q.shape[1]
    q, kk, v = q.double().repeat_interleave(rep, 1), kk.double().repeat_interleave(rep, 1), v.double()
    for t in range(q.shape[0]):
        if rule == k.MLSTM:
            f, i = sc0[t].double(), sc1[t].double()
            m_new = torch.maximum(f + m, i)
            a, b = torch.exp(f + m - m_new), torch.exp(i - m_new)
            S = a[:, None, None] * S + (b[:, None] * kk[t])[:, :, None] * v[t][:, None]
            n, m = a[:, None] * n + b[:, None] * kk[t], m_new
            low = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            out[t] = torch.einsum("hde,hd->he", S, q[t]) / low[:, None]
            continue
        kv = kk[t][:, :, None] * v[t][:, None]
        if rule == k.WKV:
            out[t] = torch.einsum("hde,hd->he", S + per_head.double()[:, :, None] * kv, q[t])
            S = w[t].double()[:, :, None] * S + kv
            continue
        S = (w[t].double()[:, :, None] if rule == k.CHANNEL else sc0[t].double()[:, None, None]) * S
        if rule == k.SSD:
            S = S + sc1[t].double()[:, None, None] * kv
            out[t] = torch.einsum("hde,hd->he", S, q[t]) + per_head.double()[:, None] * v[t]
        else:
            u = sc1[t].double()[:, None] * (v[t] - torch.einsum("hde,hd->he", S, kk[t]))
            S = S + kk[t][:, :, None] * u[:, None]
            out[t] = torch.einsum("hde,hd->he", S, q[t])
    return out, S, n, m


@pytest.mark.parametrize("rule", ["DELTA", "MLSTM", "WKV", "SSD", "CHANNEL"])
@pytest.mark.parametrize("H,G,D,E", [(4, 2, 128, 128), (2, 1, 64, 64), (3, 3, 20, 20), (2, 2, 100, 100)])
def test_chunks_agree_with_float64(rule, H, G, D, E, monkeypatch):
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda rule, rows, requests, longest, heads: requests > 0)
    rule_code = getattr(k, rule)
    if rule in ("MLSTM", "WKV"):
        G = H
    elif (H, D) == (4, 128):
        E = 40                                    # values unlike keys, no whole tiles
    for lengths in LENGTHS + ([(2048,)] if (H, D) == (4, 128) else []):
        g = torch.Generator().manual_seed(len(lengths) + D)
        T, R = sum(lengths), len(lengths)
        q, kk, v, w, sc0, sc1, per_head = _operands(rule_code, k, T, H, G, D, E, g)
        parts = [q.reshape(T, -1), kk.reshape(T, -1), v.reshape(T, -1)] + ([w.reshape(T, -1)] if w is not None else [])
        qkv = torch.cat(parts, 1).contiguous().to(DEV)
        offs = (0, G * D, 2 * G * D)
        sizes = (H * D * E, H * D, -(-H // 4) * 4)
        before = torch.randn(R, sum(sizes), generator=g) * 0.3
        results = {}
        for chunks in (True, False):
            ctx, starts, slots = _ctx(lengths, torch.bfloat16)
            state = torch.zeros(R, 4 * sum(sizes), dtype=torch.uint8, device=DEV)
            state.view(torch.float32)[slots] = before.to(DEV)
            out = torch.full((T, H * E), float("nan"), device=DEV)
            k.CHUNKS = k.STEP = chunks
            try:
                k.matrix_memory(rule_code, qkv, *offs, *(x.contiguous().to(DEV) if x is not None else None for x in (sc0, sc1)),
                                ctx, state, 0, 4 * sizes[0], 4 * (sizes[0] + sizes[1]), out, H, G, D, E,
                                w_off=2 * G * D + H * E, per_head=per_head.to(DEV).contiguous() if per_head is not None else None)
            finally:
                k.CHUNKS = k.STEP = True
            results[chunks] = out.cpu().view(T, H, E), state.view(torch.float32)[slots].cpu()
        for r in range(R):
            a, b = starts[r], starts[r + 1]
            cut = [x[a:b] if x is not None else None for x in (q, kk, v, w, sc0, sc1)]
            S0 = before[r, :sizes[0]].double().view(H, D, E)
            n0, m0 = before[r, sizes[0]:sizes[0] + sizes[1]].double().view(H, D), before[r, sum(sizes[:2]):][:H].double()
            want, S, n, m = _walk(rule_code, k, *cut, per_head, S0, n0, m0)
            errors = {}
            for chunks, (out, state) in results.items():
                off = [float((out[a:b].double() - want).norm() / want.norm()),
                       float((state[r, :sizes[0]].double().view(H, D, E) - S).norm() / S.norm())]
                if rule == "MLSTM":
                    off.append(float((state[r, sizes[0]:sizes[0] + sizes[1]].double().view(H, D) - n).norm() / n.norm()))
                    off.append(float((state[r, sum(sizes[:2]):][:H].double() - m).abs().max()) / max(1.0, float(m.abs().max())))
                errors[chunks] = off
            for got, plain in zip(errors[True], errors[False]):
                times, least = (4, 8 * ROUNDING) if rule == "MLSTM" else (2, 4 * ROUNDING)
                assert got <= max(times * plain, least), (rule, lengths, r, errors)


@pytest.mark.parametrize("rule", ["DELTA", "CHANNEL"])
@pytest.mark.parametrize("H,D,E", [(12, 128, 128), (16, 64, 72), (12, 100, 100), (3, 128, 20), (2, 36, 8)])
def test_the_delta_rules_walk_in_both_widths(rule, H, D, E, monkeypatch):
    """16 columns of the state a block (more than 74 such blocks) and 8: one chunk, part of one, whole chunks and one token
    more, against float64; the bound is the module's."""
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda rule, rows, requests, longest, heads: requests > 0)
    code, lengths = getattr(k, rule), (96, 33, 7)
    g = torch.Generator().manual_seed(H + D)
    T, R = sum(lengths), len(lengths)
    assert (R * H * -(-E // 16) > 74) == (H >= 12)
    q, kk, v, w, sc0, sc1, _ = _operands(code, k, T, H, H, D, E, g)
    on = lambda x: x.contiguous().to(DEV) if x is not None else None
    qkv = on(torch.cat([x.reshape(T, -1) for x in (q, kk, v, w) if x is not None], 1))
    before, results = torch.randn(R, H * D * E, generator=g) * 0.3, []
    for chunks in (True, False):
        monkeypatch.setattr(k, "CHUNKS", chunks)
        ctx, starts, slots = _ctx(lengths, torch.bfloat16)
        state = torch.zeros(R, H * D * E, device=DEV)
        state[slots] = before.to(DEV)
        out = torch.full((T, H * E), float("nan"), device=DEV)
        k.matrix_memory(code, qkv, 0, H * D, 2 * H * D, on(sc0), on(sc1), ctx, state.view(torch.uint8), 0, 0, 0, out, H, H, D, E,
                        w_off=2 * H * D + H * E)
        results.append((out.cpu().view(T, H, E).double(), state[slots].cpu().view(R, H, D, E).double()))
    for r in range(R):
        a, b = starts[r], starts[r + 1]
        want, S, _, _ = _walk(code, k, *[x[a:b] if x is not None else None for x in (q, kk, v, w, sc0, sc1)], None,
                              before[r].double().view(H, D, E), None, None)
        off = [[float((x - y).norm() / y.norm()) for x, y in ((o[a:b], want), (s[r], S))] for o, s in results]
        for got, plain in zip(*off):
            assert got <= max(2 * plain, 4 * ROUNDING), (lengths[r], off)


@pytest.mark.parametrize("rule", ["DELTA", "MLSTM", "WKV", "SSD", "CHANNEL"])
@pytest.mark.parametrize("space,limit", [(0, 32), (None, 64), (None, 128)])
def test_slices_have_the_bits_of_one(rule, space, limit, monkeypatch):
    """A step whose workspaces would be too large goes in slices of its portions: the same numbers in less room."""
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda rule, rows, requests, longest, heads: requests > 0)
    code, H, D, whole = getattr(k, rule), 3, 64, k.CHUNK_SPACE
    for lengths in [(1, 128, 33, 1), (300,), (129, 31, 70), (20, 64, 257)]:
        g = torch.Generator().manual_seed(len(lengths))
        T, R = sum(lengths), len(lengths)
        q, kk, v, w, sc0, sc1, per_head = _operands(code, k, T, H, H, D, D, g)
        on = lambda x: x.contiguous().to(DEV) if x is not None else None
        qkv = on(torch.cat([x.reshape(T, -1) for x in (q, kk, v, w) if x is not None], 1))
        before = torch.randn(R, H * D * D + H * D + 4, generator=g) * 0.3
        results, asked = [], []
        for cut in (False, True):
            ctx, _, _ = _ctx(lengths, torch.bfloat16)
            room = ctx.scratch
            ctx.scratch = lambda name, shape, kind: asked.append((name, tuple(shape))) or room(name, shape, kind)
            if cut and space is None:
                monkeypatch.setattr(k, "slice_tokens", lambda *a: limit)
            if cut and space is not None:
                monkeypatch.setattr(k, "CHUNK_SPACE", space)
            asked.clear()
            state = on(before).clone().view(torch.uint8)
            out = torch.full((T, H * D), float("nan"), device=DEV)
            k.matrix_memory(code, qkv, 0, H * D, 2 * H * D, on(sc0), on(sc1), ctx, state, 0, 4 * H * D * D,
                            4 * (H * D * D + H * D), out, H, H, D, D, w_off=3 * H * D, per_head=on(per_head))
            results.append((out.cpu(), state.view(torch.float32).cpu()))
        monkeypatch.undo()
        monkeypatch.setattr(k, "chunks_pay", lambda rule, rows, requests, longest, heads: requests > 0)
        assert k.CHUNK_SPACE == whole
        portions = R - (lengths[0] == 1)
        rows, (row_bytes, chunk_bytes) = min(T, portions * limit), k._space_of(code, H, D, D)
        room = 4 * dict(asked)["memory.chunks"][0]
        assert room <= rows * row_bytes + (rows // 32 + portions) * chunk_bytes + 8 * portions * H * (D + 1) + 160
        assert bool(torch.isfinite(results[0][0]).all())
        assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1]), lengths


@pytest.mark.parametrize("rule", ["DELTA", "CHANNEL", "SSD", "WKV", "MLSTM"])
def test_a_later_token_does_not_reach_an_earlier_one(rule, monkeypatch):
    """A value that is not a number stays with its own and later tokens of its own request."""
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda *a: True)
    code, H, D, lengths, at = getattr(k, rule), 2, 64, (140, 130), 45
    g = torch.Generator().manual_seed(2)
    T = sum(lengths)
    q, kk, v, w, sc0, sc1, per_head = _operands(code, k, T, H, H, D, D, g)
    outs = []
    for bad in (False, True):
        if bad:
            v[at], kk[at], q[at] = float("nan"), float("inf"), float("nan")
        qkv = torch.cat([x.reshape(T, -1) for x in (q, kk, v, w) if x is not None], 1).contiguous().to(DEV)
        ctx, _, _ = _ctx(lengths, torch.bfloat16)
        state = torch.zeros(2, 4 * (H * D * D + H * D + 4), dtype=torch.uint8, device=DEV)
        out = torch.empty(T, H * D, device=DEV)
        k.matrix_memory(code, qkv, 0, H * D, 2 * H * D, *(x.contiguous().to(DEV) if x is not None else None for x in (sc0, sc1)),
                        ctx, state, 0, 4 * H * D * D, 4 * (H * D * D + H * D), out, H, H, D, D, w_off=3 * H * D,
                        per_head=per_head.to(DEV).contiguous() if per_head is not None else None)
        outs.append(out.cpu())
    assert torch.equal(outs[0][:at], outs[1][:at]) and torch.equal(outs[0][lengths[0]:], outs[1][lengths[0]:])
    assert bool(torch.isnan(outs[1][at]).any())


@pytest.mark.parametrize("closed", [(0, 1), (0, 40), (0, 64), (31, 33), (60, 61), (0, 70)])
def test_input_gates_that_are_shut(closed, monkeypatch):
    """Log input gates of -inf, from a portion's beginning on, over whole chunks, or throughout: such tokens add
    nothing, as in the walk."""
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda *a: True)
    H, D, T, g = 2, 64, 70, torch.Generator().manual_seed(7)
    q, kk, v, w, sc0, sc1, _ = _operands(k.MLSTM, k, T, H, H, D, D, g)
    sc1[closed[0]:closed[1]] = float("-inf")
    qkv = torch.cat([x.reshape(T, -1) for x in (q, kk, v)], 1).contiguous().to(DEV)
    before = torch.randn(1, H * D * D + H * D + 4, generator=g) * 0.3
    results = []
    for chunks in (True, False):
        ctx, _, _ = _ctx((T,), torch.bfloat16)
        state, out = before.to(DEV).clone().view(torch.uint8), torch.full((T, H * D), float("nan"), device=DEV)
        monkeypatch.setattr(k, "CHUNKS", chunks)
        k.matrix_memory(k.MLSTM, qkv, 0, H * D, 2 * H * D, sc0.contiguous().to(DEV), sc1.contiguous().to(DEV), ctx, state, 0,
                        4 * H * D * D, 4 * (H * D * D + H * D), out, H, H, D, D)
        results.append((out, state.view(torch.float32)))
    for got, want in zip(*results):
        assert bool(torch.isfinite(want).all()) and bool(torch.isfinite(got).all())
        assert float((got - want).norm() / want.norm()) < 1e-5      # float32 sums of up to 70 tokens in another order


@pytest.mark.parametrize("lengths", [(70, 33), (1, 1, 1), (1, 70)])
def test_rows_off_the_wide_loads_boundaries_are_walked(lengths, monkeypatch):
    """Outputs that start on no 16-byte boundary: the chunks refuse them, and the walk's bits are the answer."""
    from crucible_b200.ops import recurrent as k
    monkeypatch.setattr(k, "chunks_pay", lambda rule, rows, requests, longest, heads: requests > 0)
    H, D, g, T, R = 2, 64, torch.Generator().manual_seed(3), sum(lengths), len(lengths)
    q, kk, v, w, sc0, sc1, per_head = _operands(k.DELTA, k, T, H, H, D, D, g)
    qkv = torch.cat([x.reshape(T, -1) for x in (q, kk, v)], 1).contiguous().to(DEV)
    qkv_off = torch.empty(qkv.numel() + 1, device=DEV)[1:].view(qkv.shape).copy_(qkv)
    outs = []
    for chunks, rows in ((True, qkv_off), (False, qkv)):
        ctx, _, _ = _ctx(lengths, torch.bfloat16)
        state = torch.zeros(R, 4 * H * D * D, dtype=torch.uint8, device=DEV)
        out = torch.full((T * H * D + 1,), float("nan"), device=DEV)[1:].view(T, H * D)
        k.CHUNKS = k.STEP = chunks
        try:
            k.matrix_memory(k.DELTA, rows, 0, H * D, 2 * H * D, sc0.contiguous().to(DEV), sc1.contiguous().to(DEV),
                            ctx, state, 0, 0, 0, out, H, H, D, D)
        finally:
            k.CHUNKS = k.STEP = True
        outs.append((out.cpu(), state.cpu()))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows_off,out_off", [(0, 1), (1, 0), (1, 1), (0, 2)])
def test_mlstm_rows_off_the_wide_boundaries(dtype, rows_off, out_off):
    """Rows or prepared rows that start on no boundary of four elements: moved one by one, the same bits."""
    from crucible_b200.ops import recurrent as k
    H, D, E, T, g = 2, 16, 24, 5, torch.Generator().manual_seed(5)
    C = H * (2 * D + E)
    proj = torch.randn(T, C + H * E, generator=g).to(dtype).to(DEV)
    gates = torch.randn(T, 2 * H, generator=g).to(DEV)
    bias = torch.randn(2, H, generator=g).to(DEV)
    results = []
    for a, b in ((0, 0), (rows_off, out_off)):
        rows = torch.empty(proj.numel() + a, dtype=dtype, device=DEV)[a:].view(proj.shape).copy_(proj)
        qkv = torch.full((T * C + b + 4,), float("nan"), device=DEV)
        keep, into = torch.empty(T, H, device=DEV), torch.empty(T, H, device=DEV)
        k.mlstm_prepare(rows, gates, bias[0], bias[1], 6.0, qkv[b:b + T * C].view(T, C), keep, into, H, D, E)
        assert bool(torch.isnan(qkv[b + T * C:]).all())
        results.append((qkv[b:b + T * C].cpu(), keep.cpu(), into.cpu()))
    assert all(torch.equal(x, y) for x, y in zip(*results))


@pytest.mark.parametrize("host", [None, "none given"])
def test_a_step_without_the_hosts_counts_is_walked(host):
    """A bfloat16 step's context that does not say what its requests bring."""
    from crucible_b200.ops import recurrent as k
    H, D, lengths, g = 2, 64, (300, 1), torch.Generator().manual_seed(4)
    T = sum(lengths)
    q, kk, v, w, sc0, sc1, _ = _operands(k.DELTA, k, T, H, H, D, D, g)
    qkv = torch.cat([x.reshape(T, -1) for x in (q, kk, v)], 1).contiguous().to(DEV)
    results = []
    for dtype in (torch.bfloat16, torch.float32):
        ctx, _, _ = _ctx(lengths, dtype)
        if dtype == torch.bfloat16:
            del ctx.host
            if host is None:
                ctx.host = None
        state, out = torch.zeros(2, 4 * H * D * D, dtype=torch.uint8, device=DEV), torch.empty(T, H * D, device=DEV)
        k.matrix_memory(k.DELTA, qkv, 0, H * D, 2 * H * D, sc0.contiguous().to(DEV), sc1.contiguous().to(DEV), ctx, state, 0, 0,
                        0, out, H, H, D, D)
        results.append((out, state))
    assert all(torch.equal(x, y) for x, y in zip(*results))
