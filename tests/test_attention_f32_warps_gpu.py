"""The 32-bit attention's blocks of 32 rows with four and with eight warps: the same bits, on both sides of the line that
chooses between them."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("H,G,D", [(6, 2, 64), (10, 1, 128), (5, 1, 192)])
@pytest.mark.parametrize("held,new,window", [(0, 33, None), (450, 31, None), (300, 130, 70)])
def test_four_and_eight_warps(H, G, D, held, new, window, monkeypatch):
    from crucible_b200 import ops
    from crucible_b200.engine.context import HostStep
    g, page, total = torch.Generator().manual_seed(D + held), 8, held + new
    per = -(-total // page)
    table = torch.randperm(per, generator=g).to(torch.int32).view(1, per).to(DEV)
    k, v = (torch.randn(per, G, page, D, generator=g).to(DEV) for _ in range(2))
    q = torch.randn(new, H * D, generator=g).to(DEV)
    ctx = SimpleNamespace(n_requests=1, req_row_start=_i32([0, new]), req_first_pos=_i32([held]),
                          host=HostStep([0], [new], [held], [total], [0]))
    outs = []
    for warps in (4, 8):
        monkeypatch.setattr(ops, "f32_attention_warps", lambda *a: warps)
        out = torch.full((new, H * D), float("nan"), device=DEV)
        assert ops.attention_f32(q, None, out, k, v, None, H, G, D, D, D ** -0.5, window, False, 0, 1.0, ctx, page, table)
        outs.append(out)
    assert torch.equal(*outs) and not torch.isnan(outs[0]).any()
