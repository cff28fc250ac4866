"""The attention of single tokens over short contexts where scores are NaN or -inf: as the split kernels, and
as float64 softmax has it, a NaN among a row's scores makes the row NaN wherever the key lies, and a row
without any weight is 0."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAN, INF = float("nan"), float("inf")


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 4, 2), (64, 8, 1), (128, 2, 2), (128, 8, 2)])
def test_nan_and_no_weight(head_dim, heads, kv_heads, plain, monkeypatch):
    from crucible_b200.engine.context import HostStep, Scratch
    from crucible_b200.ops import paged_attention, sink_attention, tensor_core as tc
    D, page = head_dim, 16
    # keys of a request, and where they are NaN: one key alone in a warp's pass, a whole pass of one warp, a
    # warp's second pass, one key among others, the first key; the query; and scores of -inf: some, all
    bad = [(33, [32], NAN), (100, range(32, 64), NAN), (600, range(512, 544), NAN), (40, [5], NAN), (1, [0], NAN),
           (50, "q", NAN), (70, range(0, 40), -INF), (45, range(45), -INF), (300, range(300), -INF), (90, [], 0.0),
           (1, [0], -INF), (64, [3], INF)]
    n, per = len(bad), 40
    g = torch.Generator().manual_seed(heads * D)
    table = torch.randperm(n * per, generator=g, dtype=torch.int32).view(n, per)
    k, v = (torch.randn(n * per, kv_heads, page, D, generator=g).bfloat16() for _ in range(2))
    q = torch.randn(n, heads * D, generator=g).abs().bfloat16()          # (positive: q k is -inf where a feature of k is)
    for r, (m, at, value) in enumerate(bad):
        if at == "q":
            q[r, 3] = value                                              # one feature of the first head's query
        else:
            for j in at:
                k[table[r, j // page].long(), :, j % page, 7] = value
    sinks = None if plain else torch.randn(heads, generator=g)
    lengths = [m for m, _, _ in bad]
    kd, vd, qd, td = (x.to(DEV) for x in (k, v, q, table))
    cache = SimpleNamespace(keys=lambda s: kd, values=lambda s: vd, page_tokens=page)
    ctx = SimpleNamespace(n_requests=n, n_tokens=n, req_row_start=_i32(list(range(n + 1))), req_first_pos=_i32([m - 1 for m in lengths]),
                          positions=_i32([m - 1 for m in lengths]), row_request=_i32(list(range(n))), block_table=lambda x: td,
                          scratch=Scratch(DEV).get, host=HostStep(list(range(n)), [1] * n, [m - 1 for m in lengths], lengths, list(range(n))))
    binding, outs = SimpleNamespace(slot=0, group=0), []
    monkeypatch.setattr(tc, "short_attention_pays", lambda *a, **kw: True)
    taken, own = [], tc.short_attention
    monkeypatch.setattr(tc, "short_attention", lambda *a, **kw: taken.append(own(*a, **kw)) or taken[-1])
    for on in (True, False):
        monkeypatch.setattr(tc, "SHORT_ATTENTION", on)
        for given in ((None,) if plain else (None, sinks.to(DEV))):
            out = torch.full((n, heads * D), 7.0, device=DEV, dtype=torch.bfloat16)
            if plain:
                paged_attention(qd, out, heads, kv_heads, D, D ** -0.5, None, ctx, cache, binding)
            else:
                sink_attention.attention(qd, None, out, given, heads, kv_heads, D, D, D ** -0.5, None, 0, 1.0, ctx, cache, binding)
            outs.append((given is not None, on, out.cpu()))
    assert taken == ([True, False] if plain else [True, True, False, False])
    for sink, on, out in outs:
        for r, (m, at, value) in enumerate(bad):
            for h in range(heads):
                j = torch.arange(m)
                kk, vv = (c[table[r, j // page].long(), h * kv_heads // heads, j % page].double() for c in (k, v))
                s = kk @ q[r, h * D:(h + 1) * D].double() * D ** -0.5
                if sink:
                    s = torch.cat([s, sinks[h:h + 1].double()])
                want = torch.softmax(s, 0)[:m] @ vv
                if bool((s == -INF).all()):
                    want = torch.zeros_like(want)
                got = out[r, h * D:(h + 1) * D].double()
                assert torch.equal(got.isnan(), want.isnan()), (r, h, sink, on)
                if not bool(want.isnan().any()):
                    # one rounding to bfloat16 (2^-9); the split kernels round their weights too
                    assert float((got - want).norm()) <= 2.0 ** -7 * float(want.norm()), (r, h, sink, on)
