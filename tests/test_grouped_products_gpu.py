"""The grouped tensor-core product at the edges of its tiles: experts of no, one, 15 to 17, 127 to 129
and many rows, every tile width that the rule can choose, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tile", [(128, 1), (128, 2), (192, 1), (256, 1)])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("counts", [(0, 1, 15, 16, 17, 0), (127, 128, 129, 0, 0, 3), (300, 0, 2, 40, 16, 1)])
def test_rows_at_the_edges_of_tiles(tile, gated, counts):
    from crucible_b200 import ops
    from crucible_b200.ops import tensor_core
    E, K, N, T = len(counts), 328, 200, sum(counts)
    g = torch.Generator().manual_seed(T)
    a = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    ops.declare_weights(w)
    rows = 128
    tiles = [(e, sum(counts[:e]) + r, min(rows, n - r)) for e, n in enumerate(counts) for r in range(0, n, rows)]
    most = len(tiles) + 3                                    # tiles beyond those in use
    plan = torch.zeros(2 + E + 3 * most, dtype=torch.int32)
    plan[0] = len(tiles)
    for i, (e, first, n) in enumerate(tiles):
        plan[2 + E + i], plan[2 + E + most + i], plan[2 + E + 2 * most + i] = e, first, n
    out = torch.full((T, N), float("nan"), dtype=torch.bfloat16 if gated else torch.float32, device=DEV)
    assert tensor_core.grouped_linear(a, w, out, plan.to(DEV), E, most, gated, tile=tile)
    at = 0
    want = torch.zeros(T, N, dtype=torch.float64)
    for e, n in enumerate(counts):
        y = a[at:at + n].cpu().double() @ w[e].cpu().double().T
        want[at:at + n] = torch.nn.functional.silu(y[:, :N]) * y[:, N:] if gated else y
        at += n
    off = (out.cpu().double() - want).abs().max() / want.abs().max()
    # float32 sums of exact products; the gated pair is rounded to bfloat16 once, its silu approximate
    assert float(off) < (6e-3 if gated else 2e-6)
