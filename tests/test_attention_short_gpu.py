"""The attention of single tokens over short contexts against float64: passes of keys and their remainders,
groups of heads, windows, sinks, gates; and its place in the dispatch."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("heads,kv_heads,page", [(1, 1, 16), (4, 2, 8), (3, 1, 16), (8, 2, 64), (10, 2, 5), (16, 2, 16)])
@pytest.mark.parametrize("window,sink,gate", [(None, False, None), (40, True, "element"), (300, False, "head"), (None, True, "element")])
def test_single_tokens_over_short_contexts(head_dim, heads, kv_heads, page, window, sink, gate, monkeypatch):
    from crucible_b200.ops import tensor_core as tc
    lengths = [1, 31, 32, 33, 255, 256, 257, 511, 513, 1030]
    n, D, per = len(lengths), head_dim, -(-1030 // page)
    g = torch.Generator().manual_seed(heads * head_dim + page)
    table = torch.randperm(n * per, generator=g, dtype=torch.int32).view(n, per)
    k, v = (torch.randn(n * per, kv_heads, page, D, generator=g).bfloat16() for _ in range(2))
    q = torch.randn(n, heads * D, generator=g).bfloat16()
    logit = torch.randn(n, heads * (D if gate == "element" else 1), generator=g).bfloat16() if gate else None
    sinks = torch.randn(heads, generator=g) if sink else None
    scale, out_scale = D ** -0.5, 0.75
    given = table.clone()
    if window:                                    # pages behind the window were given back
        for r, m in enumerate(lengths):
            given[r, :max(0, m - window) // page] = -1
    monkeypatch.setattr(tc, "short_attention_pays", lambda *a: True)
    ctx = SimpleNamespace(req_row_start=_i32(list(range(n + 1))), req_first_pos=_i32([m - 1 for m in lengths]))
    out = torch.full((n, heads * D + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    assert tc.short_attention(q.to(DEV), out[:, :heads * D], k.to(DEV), v.to(DEV), ctx, given.to(DEV), n, 1280, heads, kv_heads, D,
                              scale, window, page, sinks.to(DEV) if sink else None, out_scale,
                              logit.to(DEV) if gate else None, gate == "head")
    for r, m in enumerate(lengths):
        at = torch.arange(max(0, m - window) if window else 0, m)
        for h in range(heads):
            kk, vv = (c[table[r, at // page].long(), h * kv_heads // heads, at % page].double() for c in (k, v))
            s = kk @ q[r, h * D:(h + 1) * D].double() * scale
            if sink:
                s = torch.cat([s, sinks[h:h + 1].double()])
            want = torch.softmax(s, 0)[:len(at)] @ vv * out_scale
            if gate:
                want = want * torch.sigmoid(logit[r, h * D:(h + 1) * D].double() if gate == "element" else logit[r, h].double())
            got = out[r, h * D:(h + 1) * D].cpu().double()
            # one rounding to bfloat16 (2^-9); scores and sums in fp32, ex2.approx (2^-22)
            assert float((got - want).norm() / want.norm()) < 2.0 ** -8
    assert bool((out[:, heads * D:] == 7.0).all())


def test_both_dispatches_take_it(monkeypatch):
    from crucible_b200.engine.context import HostStep, Scratch
    from crucible_b200.ops import paged_attention, sink_attention, tensor_core as tc
    n, G, H, D, page = 5, 2, 8, 64, 16
    g = torch.Generator().manual_seed(3)
    lengths = [7, 200, 100, 256, 31]
    table = torch.randperm(n * 16, generator=g, dtype=torch.int32).view(n, 16).to(DEV)
    k, v = (torch.randn(n * 16, G, page, D, generator=g).to(DEV).bfloat16() for _ in range(2))
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    q = torch.randn(n, H * D, generator=g).to(DEV).bfloat16()
    ctx = SimpleNamespace(n_requests=n, n_tokens=n, req_row_start=_i32(list(range(n + 1))), req_first_pos=_i32([m - 1 for m in lengths]),
                          positions=_i32([m - 1 for m in lengths]), row_request=_i32(list(range(n))), block_table=lambda x: table,
                          scratch=Scratch(DEV).get, host=HostStep(list(range(n)), [1] * n, [m - 1 for m in lengths], lengths, list(range(n))))
    binding, sinks = SimpleNamespace(slot=0, group=0), torch.randn(H, generator=g).to(DEV)
    calls, own = [], tc.short_attention
    monkeypatch.setattr(tc, "short_attention", lambda *a, **kw: calls.append(own(*a, **kw)) or calls[-1])
    outs = []
    for on in (True, False):
        monkeypatch.setattr(tc, "SHORT_ATTENTION", on)
        a, b = (torch.empty(n, H * D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
        paged_attention(q, a, H, G, D, D ** -0.5, None, ctx, cache, binding)
        sink_attention.attention(q, None, b, sinks, H, G, D, D, D ** -0.5, None, 0, 1.0, ctx, cache, binding)
        outs.append((a, b))
    assert calls == [True, True, False, False]
    for x, y in zip(*outs):                       # (the split kernels round their weights to bfloat16)
        assert float((x.float() - y.float()).norm() / y.float().norm()) < 2.0 ** -7
