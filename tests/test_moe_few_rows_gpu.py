"""Steps of few tokens through a mixture of experts: the weight rows of the chosen experts dealt over the
blocks, and a plain shared expert that rides with them, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,k,used,most", [(1, 8, 1, 1), (65, 256, 3, 9), (200, 264, 5, 5), (2816, 128, 2, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gated", [False, True])
def test_weight_rows_over_the_blocks(n, k, used, most, dtype, gated):
    from crucible_b200.ops import moe
    g = torch.Generator().manual_seed(n + used)
    rows = [1 + (5 * i) % 7 for i in range(used)]
    pairs, experts = sum(rows), [most - 1 - i for i in range(used)]
    plan = torch.full((2 + most + 3 * (most + 2),), 1 << 20, dtype=torch.int32)
    plan[0] = used
    for i, e in enumerate(experts):
        for j, v in enumerate((e, sum(rows[:i]), rows[i])):
            plan[2 + most + j * (most + 2) + i] = v
    order = torch.randperm(pairs, generator=g, dtype=torch.int32)
    weight = torch.rand(pairs, generator=g) + 0.5
    a = torch.randn(pairs, k, generator=g).to(dtype)
    w = (torch.randn(most, (2 if gated else 1) * n, k, generator=g) * k ** -0.5).to(dtype)
    out = torch.full((pairs, n), 7.0, dtype=dtype if gated else torch.float32, device=DEV)
    assert moe.expert_rows_small(gated, a.to(DEV), w.to(DEV), n, plan.to(DEV), most, most + 2, order.to(DEV), 1,
                                 weight.to(DEV), out)
    want, at = torch.zeros(pairs, n, dtype=torch.float64), 0
    for e, r in zip(experts, rows):
        for s in range(at, at + r):
            p = int(order[s])
            y = w[e].double() @ (a[p] if gated else a[s]).double()
            if gated:
                want[s] = y[:n] / (1 + torch.exp(-y[:n])) * y[n:]
            else:
                want[p] = y * float(weight[p])
        at += r
    # fp32 sums over k; bfloat16 results are rounded once (2^-9)
    assert float((out.cpu().double() - want).norm() / want.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 and gated else 2e-6)


@pytest.mark.parametrize("tokens", [1, 2, 3, 7, 127, 128, 129])
@pytest.mark.parametrize("shared", [520, 1024, 600])
def test_a_plain_shared_expert_rides(tokens, shared, monkeypatch):
    from crucible_b200.config.model_config import FeedForwardSpec
    from crucible_b200.engine.context import Scratch
    from crucible_b200.parts import FEED_FORWARDS
    from crucible_b200.parts.moe import MixtureOfExperts
    from types import SimpleNamespace
    monkeypatch.setattr(MixtureOfExperts, "SORTED_MIN_PAIRS", ((0, 4),))
    d, f, E, top = 256, 520, 5, 2
    part = FEED_FORWARDS.build("moe", FeedForwardSpec("moe", d, f, (("experts", E), ("top", top), ("shared_intermediate", shared))))
    g = torch.Generator().manual_seed(tokens)
    w = {t.name: (torch.randn(t.shape, generator=g) * t.shape[-1] ** -0.5).to(DEV).bfloat16() for t in part.tensors()}
    part.bind(w, torch.bfloat16, torch.device(DEV))
    assert part.slices == {520: 1, 1024: 2, 600: 0}[shared]       # (600 would be padded by too much)
    h = torch.randn(tokens, d, generator=g).to(DEV).bfloat16()
    x = torch.randn(tokens, d, generator=g).to(DEV)
    got = x.clone()
    part.forward(SimpleNamespace(scratch=Scratch(DEV).get, announce_norm=None, norm_ahead=lambda rows: None), h, got)
    hd, w = h.double(), {k: v.double() for k, v in w.items()}
    ffn = lambda y, p: ((lambda z: z / (1 + torch.exp(-z)))(y @ w[p + "gate"].T) * (y @ w[p + "up"].T)) @ w[p + "down"].T
    z = hd @ w["router"].T
    best, idx = z.topk(top, 1)
    want = x.double() + ffn(hd, "shared.")
    for t in range(tokens):
        for p, e in zip(torch.softmax(best[t], 0), idx[t]):
            want[t] += p * ffn(hd[t:t + 1], f"e{int(e)}.")[0]
    # activations of the pairs are rounded to bfloat16 (2^-9 each, summed over f with random signs)
    assert float((got.double() - want).norm() / (want - x.double()).norm()) < 2.0 ** -7
