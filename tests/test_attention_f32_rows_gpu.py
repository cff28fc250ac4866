"""The 32-bit attention with few blocks (eight warps to 32 rows) and with many (four): a request's rows have the same
bits alone and beside others, for contexts that end inside a tile, windows, chunks and kept first tokens."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,D,window,keep,chunked", [
    (6, 2, 64, None, 0, False), (4, 1, 64, 70, 5, False), (8, 2, 128, None, 0, False), (2, 2, 128, 100, 0, True),
    (3, 1, 192, 90, 33, False), (5, 1, 40, None, 0, False)])
def test_alone_and_beside_others(H, G, D, window, keep, chunked):
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention
    g, page = torch.Generator().manual_seed(D + H), 8
    every = [(0, 33), (200, 41), (63, 1), (5, 130)] + [(7 * i, 97) for i in range(24)]
    R = len(every)
    per = -(-max(h + n for h, n in every) // page)
    table = torch.randperm(R * per, generator=g).to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per, G, page, D, generator=g).to(DEV)
    v = torch.randn(R * per, G, page, D, generator=g).to(DEV)
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    starts = [0]
    for _, n in every:
        starts.append(starts[-1] + n)
    q = torch.randn(starts[-1], H * D, generator=g).to(DEV)

    def run(which):
        held, counts = [every[r][0] for r in which], [every[r][1] for r in which]
        contexts, at = [h + n for h, n in zip(held, counts)], [0]
        for n in counts:
            at.append(at[-1] + n)
        rows = torch.cat([q[starts[r]:starts[r + 1]] for r in which])
        mine = table[which].contiguous()
        ctx = SimpleNamespace(n_requests=len(which), n_tokens=at[-1], req_row_start=_i32(at), req_first_pos=_i32(held),
                              positions=_i32([h + i for h, n in zip(held, counts) for i in range(n)]),
                              row_request=_i32([r for r, n in enumerate(counts) for _ in range(n)]),
                              block_table=lambda group: mine,
                              host=HostStep(list(range(len(which))), counts, held, contexts, list(range(len(which)))))
        out = torch.full((at[-1], H * D), float("nan"), device=DEV)
        sink_attention.attention(rows, None, out, None, H, G, D, D, D ** -0.5, window, keep, 1.0, ctx, cache,
                                 SimpleNamespace(slot=0, group=0), chunked=chunked)
        return out
    together = run(list(range(R)))
    assert not torch.isnan(together).any()
    for r in (0, 1, 2, 3, 9):
        assert torch.equal(run([r]), together[starts[r]:starts[r + 1]])
    # and against plain attention in 64 bits: one request whole
    r, (held, n) = 1, every[1]
    places = table[r].long().repeat_interleave(page) * page + torch.arange(per * page, device=DEV) % page
    pos, key = held + torch.arange(n, device=DEV)[:, None], torch.arange(held + n, device=DEV)[None]
    low = torch.zeros_like(pos) if window is None else pos - pos % window if chunked else pos - window + 1
    seen = (key <= pos) & ((key >= low) | (key < keep))
    for h in range(H):
        kk, vv = (t.permute(0, 2, 1, 3).reshape(-1, G, D)[places[:held + n], h * G // H].double() for t in (k, v))
        s = (q[starts[r]:starts[r + 1], h * D:(h + 1) * D].double() @ kk.T * D ** -0.5).masked_fill(~seen, float("-inf"))
        want = torch.softmax(s, -1) @ vv
        got = together[starts[r]:starts[r + 1], h * D:(h + 1) * D].double()
        assert float((got - want).abs().max() / want.abs().max()) < 2e-6        # sums of 241 float32 products, 2^-24 each
