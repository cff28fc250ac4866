"""The prompt attention's gate by itself: with a window of one token a row's softmax has one weight, 1, and with values of 1
a result is sigmoid(logit), for every logit that bfloat16 has."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("D,H,G", [(64, 4, 4), (128, 16, 2), (256, 8, 1), (64, 48, 1), (128, 40, 1)])
@pytest.mark.parametrize("per_head", [False, True])
def test_every_logit_to_the_results_rounding(D, H, G, per_head):
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import sink_attention, tensor_core
    page, rows = 16, 65536 // (H if per_head else H * D) + 1
    rows = max(rows, 64)                                          # (fewer packed rows are another kernel's)
    pages = -(-rows // page)
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1)
    ones = torch.ones((pages, G, page, D), dtype=torch.bfloat16, device=DEV)
    cache = SimpleNamespace(keys=lambda s: ones, values=lambda s: ones, page_tokens=page)
    ctx = SimpleNamespace(n_requests=1, n_tokens=rows, req_row_start=_i32([0, rows]), req_first_pos=_i32([0]),
                          positions=_i32(list(range(rows))), row_request=_i32([0] * rows), block_table=lambda group: table,
                          host=HostStep([0], [rows], [0], [rows], [0]))
    bits = torch.arange(rows * (H if per_head else H * D), dtype=torch.int64) % 65536
    logits = (bits - 65536 * (bits > 32767)).to(torch.int16).view(torch.bfloat16).view(rows, -1)
    q = torch.zeros(rows, H * D, dtype=torch.bfloat16, device=DEV)
    out = torch.full_like(q, float("nan"))
    reached = []
    real = tensor_core._attention_tcgen05
    tensor_core._attention_tcgen05 = lambda *a, **k: reached.append(real(*a, **k)) or reached[-1]
    try:
        sink_attention.attention(q, logits.to(DEV), out, None, H, G, D, D, D ** -0.5, 1, 0, 1.0, ctx, cache,
                                 SimpleNamespace(slot=0, group=0), gate_per_head=per_head)
    finally:
        tensor_core._attention_tcgen05 = real
    torch.cuda.synchronize()
    tensor_core.check_status(DEV)
    assert reached == [True]
    x = logits.double()
    if per_head:
        x = x.repeat_interleave(D, 1)
    want = torch.where(x < 0, torch.exp(x), torch.ones_like(x)) / (1 + torch.exp(-x.abs()))
    got, nan = out.cpu().double(), torch.isnan(x)
    assert torch.equal(torch.isnan(got), nan)
    # half of bfloat16's spacing at the true value (8 bits, down to 2^-133), and the gate's own error in 32 bits: a unit of
    # expf, half of the sum's, two of the division, half of the product's, 2^-23 each: under 2^-20 of the value
    half = torch.clamp(torch.exp2(torch.floor(torch.log2(want.clamp(min=2.0 ** -140))) - 8), min=2.0 ** -134)
    assert bool(((got - want).abs() <= half + want * 2.0 ** -20)[~nan].all())
