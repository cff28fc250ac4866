"""Two products of the same rows in one launch, bfloat16 and float32 results, against float64 and against
the two launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 33, 128, 129, 300, 1100])
@pytest.mark.parametrize("n_main,n_second,k", [(64, 4, 64), (320, 16, 136), (1024, 32, 72), (2560, 8, 256), (448, 260, 1032),
                                               (128, 5, 64)])
def test_two_products_in_one(m, n_main, n_second, k):
    from crucible_b200 import ops
    from crucible_b200.ops import tensor_core
    g = torch.Generator().manual_seed(m + n_main)
    a = torch.randn(m, k, generator=g).to(DEV).bfloat16()
    w = (torch.randn(n_main + n_second, k, generator=g) * k ** -0.5).to(DEV).bfloat16()
    ops.declare_weights(w)
    out = torch.full((m, n_main + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    second = torch.full((m, n_second), 7.0, device=DEV)
    before = ops.LAUNCHES[0]
    ops.linear_split(a, w, w[:n_main], w[n_main:], out[:, :n_main], second)
    launches = ops.LAUNCHES[0] - before
    want = a.double() @ w.double().T
    # a rounding of the result (2^-9) beside fp32 sums over k
    assert float((out[:, :n_main].double() - want[:, :n_main]).norm() / want[:, :n_main].norm()) < 2.0 ** -8
    assert float((second.double() - want[:, n_main:]).norm() / want[:, n_main:].norm()) < 2e-6
    assert bool((out[:, n_main:] == 7.0).all())
    assert launches == (2 if n_second % 4 and m > 16 else 1)
    tensor_core.check_status(DEV)


@pytest.mark.parametrize("tile", [(64, 1), (128, 1), (192, 1), (256, 1), (256, 0)])
def test_every_tile_and_shares_of_k(tile, monkeypatch):
    from crucible_b200.ops import tensor_core as tc
    for m, n_main, n_second, k, shares in ((130, 704, 36, 328, 1), (40, 192, 68, 520, 3 if tile[1] else 1)):
        g = torch.Generator().manual_seed(m)
        a = torch.randn(m, k, generator=g).to(DEV).bfloat16()
        w = (torch.randn(n_main + n_second, k, generator=g) * k ** -0.5).to(DEV).bfloat16()
        monkeypatch.setattr(tc, "_split_tile", lambda *_: tile)
        monkeypatch.setattr(tc, "k_splits", lambda *_: shares)
        out = torch.empty(m, n_main, device=DEV, dtype=torch.bfloat16)
        second = torch.full((m + 1, n_second), 7.0, device=DEV)
        assert tc.linear_split(a, w, out, second[:m])
        want = a.double() @ w.double().T
        assert float((out.double() - want[:, :n_main]).norm() / want[:, :n_main].norm()) < 2.0 ** -8
        assert float((second[:m].double() - want[:, n_main:]).norm() / want[:, n_main:].norm()) < 2e-6
        assert bool((second[m] == 7.0).all())
        tc.check_status(DEV)
