"""Float32 results by a long K whose narrowest tiles leave no room for two shares of K: the choice, and the products
against float64."""
import pytest
import torch


def test_wider_tiles_where_two_shares_then_fit():
    from crucible_b200.ops import tensor_core as tc
    choice = lambda m, n, k, epi=tc.ACCUM_F32: tc._tile_and_shares(m, n, k, epi)
    for m, n, k, epi in ((256, 2048, 5632, tc.ACCUM_F32),        # two shares of 64 columns fit
                         (257, 2048, 3520, tc.ACCUM_F32),        # the chain is short
                         (385, 2048, 4096, tc.ACCUM_F32),        # 128 columns, and a chain too short for them
                         (513, 2048, 8192, tc.ACCUM_F32),        # no room for two shares
                         (257, 2048, 5632, tc.STORE_BF16)):
        assert choice(m, n, k, epi) == tc._tile_width(m, n, epi)
    assert choice(257, 2048, 3584) == (96, 1, 2)
    assert choice(384, 2048, 8192, tc.STORE_F32) == (96, 1, 2)
    assert choice(385, 2048, 5632) == choice(512, 2048, 5120) == (128, 1, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(257, 2048, 3584), (384, 2044, 4104), (385, 2048, 5632), (512, 2044, 5128),
                                   (640, 1024, 4096)])
def test_products_in_two_wide_shares(m, n, k):
    from crucible_b200.ops import tensor_core as tc
    dev = "cuda:0"
    assert tc._tile_and_shares(m, n, k, tc.ACCUM_F32)[2:] == (2,)
    g = torch.Generator().manual_seed(m)
    a = torch.randn(m, k, generator=g).to(dev).bfloat16()
    w = (torch.randn(n, k, generator=g) * k ** -0.5).to(dev).bfloat16()
    base = torch.randn(m, n, generator=g).to(dev)
    want = a.double() @ w.double().T
    out = torch.full((m + 1, n), 7.0, device=dev)
    assert tc.linear(a, w, out[:m])
    # fp32 sums over k
    assert float((out[:m].double() - want).norm() / want.norm()) < 4e-6
    assert bool((out[m] == 7.0).all())
    # the sum, and what the next norm reads
    gain = torch.rand(n, generator=g).to(dev) + 0.5
    emit = tc.NormEmit(gain, torch.empty(m, n, device=dev, dtype=torch.bfloat16), torch.zeros(-(-n // 32), m, device=dev))
    acc = base.clone()
    assert tc.linear(a, w, acc, accumulate=True, emit=emit)
    want += base.double()
    assert float((acc.double() - want).norm() / want.norm()) < 4e-6
    if n % 32 == 0:
        assert emit.parts == -(-n // tc._tile_and_shares(m, n, k, tc.ACCUM_F32)[0])
        assert torch.equal(emit.scaled, (acc * gain).bfloat16())
        squares = emit.sumsq[:emit.parts].double().sum(0)
        assert float((squares / acc.double().square().sum(1) - 1).abs().max()) < 1e-5
    else:
        assert emit.parts is None
    tc.check_status(dev)
