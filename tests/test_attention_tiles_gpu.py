"""The tcgen05 prompt attention over group sizes that do and do not divide a tile's 128 rows, from one tile of
keys to more than its ring holds, with and without gates: every row against the CUDA-core kernel."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,D,window,gate", [
    (3, 1, 64, None, "element"), (8, 8, 64, 130, "head"), (24, 1, 64, None, "element"),
    (48, 1, 64, None, "element"), (144, 1, 64, None, "head"),      # rows fetched by hand: 96 of 128; two tiles a token
    (10, 2, 128, None, "element"), (4, 4, 128, 200, None), (40, 1, 128, None, "element"),
    (7, 1, 256, None, "element"), (16, 1, 256, 300, None), (48, 1, 256, None, "head")])
@pytest.mark.parametrize("requests", [
    [(0, 65)], [(63, 65), (0, 128)], [(250, 70), (0, 200), (511, 90)], [(1100, 130), (0, 70)]])
def test_every_group_size_and_number_of_tiles(H, G, D, window, gate, requests):
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention, tensor_core
    g, page, R = torch.Generator().manual_seed(H + D), 16, len(requests)
    held, counts = [h for h, _ in requests], [n for _, n in requests]
    contexts, T = [h + n for h, n in requests], sum(counts)
    per = -(-max(contexts) // page)
    table = torch.randperm(R * per, generator=g) if H % 3 else torch.arange(R * per)     # scattered pages, or runs
    table = table.to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per, G, page, D, generator=g).to(torch.bfloat16).to(DEV)
    v = k if D == 256 else torch.randn(k.shape, generator=g).to(torch.bfloat16).to(DEV)
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(held),
                          positions=_i32([h + i for h, n in requests for i in range(n)]),
                          row_request=_i32([r for r, n in enumerate(counts) for _ in range(n)]),
                          block_table=lambda group: table, host=HostStep(list(range(R)), counts, held, contexts, list(range(R))))
    wide = torch.full((T, 2 * H * D + 8), float("nan"), dtype=torch.bfloat16, device=DEV)  # rows inside wider ones
    q = wide[:, 8:8 + H * D]
    q.copy_(torch.randn(T, H * D, generator=g) * 3.0)             # (scores that raise the running maximum)
    logits = None
    if gate == "element":
        logits = wide[:, 8 + H * D:]
        logits.copy_(torch.randn(T, H * D, generator=g) * 4.0)
        logits[0, :4] = torch.tensor([float("inf"), -float("inf"), -120.0, 90.0])
    elif gate == "head":
        logits = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    sinks = torch.randn(H, generator=g).to(DEV)
    outs = []
    for use in (True, False):
        sink_attention.TENSOR_CORES = use
        try:
            out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
            sink_attention.attention(q, logits, out, sinks, H, G, D, D, D ** -0.5, window, 0, 1.0, ctx, cache,
                                     SimpleNamespace(slot=0, group=0), gate_per_head=gate == "head")
        finally:
            sink_attention.TENSOR_CORES = True
        outs.append(out.float())
    torch.cuda.synchronize()
    tensor_core.check_status(DEV)
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err < 1.5e-2                                        # both round P and the result to bfloat16 (2^-8)


@pytest.mark.parametrize("H,window", [(16, None), (8, 300), (7, None), (48, None)])       # (the last: rows fetched by hand)
@pytest.mark.parametrize("cols", [192, 64])
@pytest.mark.parametrize("requests", [[(0, 65)], [(127, 65), (0, 20)], [(300, 90), (0, 130), (383, 129)], [(1500, 140)]])
def test_latent_rows_of_which_some_features_are_values(H, window, cols, requests):
    """Rows of 256 that are keys and values at once, read up to `cols` features: those as the CUDA-core kernel has
    them, from one tile of keys to more than the ring holds."""
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention, tensor_core
    g, page, R, D = torch.Generator().manual_seed(H + cols), 16, len(requests), 256
    held, counts = [h for h, _ in requests], [n for _, n in requests]
    contexts, T = [h + n for h, n in requests], sum(counts)
    per = -(-max(contexts) // page)
    table = (torch.randperm(R * per, generator=g) if H % 3 else torch.arange(R * per)).to(torch.int32).view(R, per).to(DEV)
    k = torch.randn(R * per, 1, page, D, generator=g).to(torch.bfloat16).to(DEV)
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: k, page_tokens=page)
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_first_pos=_i32(held),
                          positions=_i32([h + i for h, n in requests for i in range(n)]),
                          row_request=_i32([r for r, n in enumerate(counts) for _ in range(n)]),
                          block_table=lambda group: table, host=HostStep(list(range(R)), counts, held, contexts, list(range(R))))
    q = (torch.randn(T, H * D, generator=g) * 3.0).to(torch.bfloat16).to(DEV)
    outs = []
    for use in (True, False):
        sink_attention.TENSOR_CORES = use
        try:
            out = torch.full((T, H * D), float("nan"), dtype=torch.bfloat16, device=DEV)
            sink_attention.attention(q, None, out, None, H, 1, D, D, D ** -0.5, window, 0, 1.0, ctx, cache,
                                     SimpleNamespace(slot=0, group=0), value_cols=cols)
        finally:
            sink_attention.TENSOR_CORES = True
        outs.append(out.view(T, H, D)[..., :cols].float())
    torch.cuda.synchronize()
    tensor_core.check_status(DEV)
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err < 1.5e-2                                        # both round P and the result to bfloat16 (2^-8)
