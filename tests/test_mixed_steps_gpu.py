"""A step of decoded tokens beside a prompt's portion on the tcgen05 attention, the decoded tokens with it
or in a launch of their own: every row against the CUDA-core kernel on the same inputs."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,D,window,keep,chunked,gate", [
    (8, 2, 128, 100, 8, False, "element"), (4, 4, 64, None, 0, False, "head"), (6, 2, 64, 96, 0, True, None),
    (16, 1, 256, None, 0, False, None)])            # the last: rows that are keys and values at once
@pytest.mark.parametrize("apart", [False, True])
@pytest.mark.parametrize("singles,portion", [([200], 65), ([1, 130, 257], 64), ([60] * 20, 130)])
def test_decoded_tokens_beside_a_portion(H, G, D, window, keep, chunked, gate, singles, portion, apart,
                                          monkeypatch):
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention, tensor_core
    g = torch.Generator().manual_seed(H + len(singles))
    contexts, page = singles + [portion + 37], 16
    per = -(-max(contexts) // page)
    R = len(contexts)
    table = torch.randperm(R * per, generator=g).to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per + 1, G, page, D, generator=g).to(torch.bfloat16).to(DEV)
    v = k if D == 256 else torch.randn(k.shape, generator=g).to(torch.bfloat16).to(DEV)
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    counts = [1] * len(singles) + [portion]
    firsts = [c - n for c, n in zip(contexts, counts)]
    T = sum(counts)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    host = HostStep(list(range(R)), counts, firsts, contexts, list(range(R)))
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(firsts),
                          positions=_i32([f + i for f, n in zip(firsts, counts) for i in range(n)]),
                          row_request=_i32([r for r, n in enumerate(counts) for _ in range(n)]),
                          block_table=lambda group: table, host=host,
                          scratch=lambda name, shape, dtype: torch.full(tuple(shape), float("nan"), dtype=dtype, device=DEV))
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16).to(DEV)
    logits = None if gate is None else torch.randn(T, H * D if gate == "element" else H, generator=g).to(torch.bfloat16).to(DEV)
    sinks = torch.randn(H, generator=g).to(DEV)
    seen, real = [], tensor_core._attention_tcgen05

    def spy(*a, **kw):
        seen.append(a[4].count)
        return real(*a, **kw)
    monkeypatch.setattr(tensor_core, "_attention_tcgen05", spy)
    if apart:
        monkeypatch.setattr(tensor_core, "MIXED_REACH", 0)
    outs = []
    for use in (True, False):
        monkeypatch.setattr(sink_attention, "TENSOR_CORES", use)
        out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        sink_attention.attention(q, logits, out, sinks, H, G, D, D, D ** -0.5, window, keep, 0.8, ctx, cache,
                                 SimpleNamespace(slot=0, group=0), gate_per_head=gate == "head", chunked=chunked)
        outs.append(out.float())
    assert seen == [1 if apart else R]                         # the portion alone, or the step
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err < 1.5e-2                                        # both round P and the result to bfloat16 (2^-8)


@pytest.mark.parametrize("H,G,D", [(8, 2, 128), (4, 4, 64), (16, 1, 256), (144, 1, 64)])      # (the last: two tiles a token)
@pytest.mark.parametrize("singles,portions", [(1, [200, 65, 70]), (3, [130, 70, 65]), (7, [64, 300, 65]), (20, [400])])
def test_tokens_beside_several_portions_have_a_tile_each(H, G, D, singles, portions):
    """Fewer, as many and more single tokens than portions: every one of the step's rows is written, with
    the values of the CUDA-core kernel."""
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention
    g, page = torch.Generator().manual_seed(H + singles), 16
    counts = [1] * singles + portions
    held = [(37 * i) % 150 for i in range(singles)] + [0, 41, 130][:len(portions)]
    R, T, contexts = len(counts), sum(counts), [c + h for c, h in zip(counts, held)]
    per = -(-max(contexts) // page)
    table = torch.randperm(R * per, generator=g).to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per, G, page, D, generator=g).to(torch.bfloat16).to(DEV)
    v = k if D == 256 else torch.randn(k.shape, generator=g).to(torch.bfloat16).to(DEV)
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(held),
                          positions=_i32([h + i for h, n in zip(held, counts) for i in range(n)]),
                          row_request=_i32([r for r, n in enumerate(counts) for _ in range(n)]),
                          block_table=lambda group: table, host=HostStep(list(range(R)), counts, held, contexts, list(range(R))))
    assert ctx.host.lead_single == singles
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16).to(DEV)
    outs = []
    for use in (True, False):
        sink_attention.TENSOR_CORES = use
        try:
            out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
            sink_attention.attention(q, None, out, None, H, G, D, D, D ** -0.5, None, 0, 1.0, ctx, cache,
                                     SimpleNamespace(slot=0, group=0))
        finally:
            sink_attention.TENSOR_CORES = True
        outs.append(out.float())
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err < 1.5e-2                                        # both round P and the result to bfloat16 (2^-8)


@pytest.mark.parametrize("counts,held,window,keep,ordered", [
    ([64, 65], [0, 0], None, 0, True),              # one and two tiles of keys: a group without any, a tile each
    ([300], [85], None, 0, False),                  # three, scattered pages
    ([130, 500, 3], [126, 600, 1500], None, 0, True),       # four to nine, one copy a tile
    ([900], [0], 130, 0, False),                    # tiles that a window leaves
    ([400], [700], 100, 200, True)])                # the kept first tokens' tiles come first
def test_heads_of_128_two_groups_of_softmax_warps(counts, held, window, keep, ordered):
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import tensor_core
    H, G, D, page, R, T = 4, 2, 128, 16, len(counts), sum(counts)
    g = torch.Generator().manual_seed(T)
    per = -(-max(c + h for c, h in zip(counts, held)) // page)
    table = (torch.arange(R * per) if ordered else torch.randperm(R * per, generator=g)).to(torch.int32).view(R, per)
    k, v = (torch.randn(R * per + 1, G, page, D, generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    host = HostStep(list(range(R)), counts, held, [c + h for c, h in zip(counts, held)], list(range(R)))
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(held), host=host)
    whole = tensor_core._Requests(ctx, table.to(DEV), 0, R, max(counts), host.context_bucket, T)
    out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert tensor_core._attention_tcgen05(q.to(DEV), out, k.to(DEV), v.to(DEV), whole, H, G, D, D ** -0.5, window,
                                          SimpleNamespace(page_tokens=page), keep_first=keep)
    for r in range(R):
        n, total = counts[r], counts[r] + held[r]
        keys, vals = (x[table[r].long()].transpose(0, 1).reshape(G, -1, D)[:, :total].double() for x in (k, v))
        s = torch.einsum("nghd,gkd->nghk", q[starts[r]:starts[r + 1]].double().view(n, G, H // G, D), keys) * D ** -0.5
        at, key = torch.arange(held[r], total)[:, None], torch.arange(total)[None]
        seen = (key <= at) & ((key > at - window) | (key < keep) if window else True)
        p = torch.softmax(s.masked_fill(~seen[:, None, None], -torch.inf), -1)
        want = torch.einsum("nghk,gkd->nghd", p, vals).reshape(n, -1)
        err = (out[starts[r]:starts[r + 1]].double().cpu() - want).abs().max() / want.abs().max()
        assert float(err) < 1.5e-2                              # P and the result rounded to bfloat16 (2^-8 each)


@pytest.mark.parametrize("H,G,D", [(4, 4, 64), (8, 2, 128), (16, 1, 256)])
@pytest.mark.parametrize("counts,held", [([65, 130], [0, 37]), ([1, 1, 300], [40, 200, 11])])
def test_a_logit_a_head_counts_before_the_rounding(H, G, D, counts, held):
    """The tiles' gate of one logit a head: the bits of a gate with that logit at each of the head's features,
    which is multiplied in before the result is rounded to bfloat16."""
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention
    g, page, R, T = torch.Generator().manual_seed(D), 16, len(counts), sum(counts)
    contexts = [c + h for c, h in zip(counts, held)]
    per = -(-max(contexts) // page)
    table = torch.randperm(R * per, generator=g).to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per, G, page, D, generator=g).to(torch.bfloat16).to(DEV)
    v = k if D == 256 else torch.randn(k.shape, generator=g).to(torch.bfloat16).to(DEV)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(held),
                          block_table=lambda group: table, host=HostStep(list(range(R)), counts, held, contexts, list(range(R))))
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    q = torch.randn(T, H * D, generator=g).to(torch.bfloat16).to(DEV)
    rows = torch.randn(T, H + 3, generator=g).to(torch.bfloat16).to(DEV)      # columns of a wider projection
    outs = []
    for per_head in (True, False):
        gate = rows[:, 1:H + 1] if per_head else rows[:, 1:H + 1].repeat_interleave(D, 1).contiguous()
        out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        sink_attention.attention(q, gate, out, None, H, G, D, D, D ** -0.5, None, 0, 1.0, ctx, cache,
                                 SimpleNamespace(slot=0, group=0), gate_per_head=per_head)
        outs.append(out)
    assert torch.equal(*outs) and bool(torch.isfinite(outs[0]).all())
