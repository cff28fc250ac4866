"""The tensor-core product with one block an SM over the tiles, against float64: edges of its tiles, more
tiles than SMs (both accumulators in turn), every epilogue and form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(m, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn(m, k, generator=g).to(DEV).bfloat16()
    w = (torch.randn(n, k, generator=g) * k ** -0.5).to(DEV).bfloat16()
    return a, w, a.double() @ w.double().T


def _close(got, want, bits):
    # one rounding of the result (2^-9 for bfloat16) and a sum over k in fp32
    return float((got.double() - want).norm() / want.norm()) < 2.0 ** -bits


def _gated(p):
    g, u = p.chunk(2, 1)
    return g / (1 + torch.exp(-g)) * u


@pytest.mark.parametrize("bn", [128, 192, 256])
@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (127, 256, 8), (129, 264, 200), (2050, 2568, 136), (4100, 776, 328)])
def test_products_in_waves(m, n, k, bn):
    from crucible_b200.ops import tensor_core as tc
    a, w, want = _inputs(m, n, k, m + n)
    out = torch.full((m, n + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    assert tc._gemm_waves(a, w, out[:, :n], n, tc.STORE_BF16, bn)
    assert _close(out[:, :n], want, 8) and bool((out[:, n:] == 7.0).all())
    assert tc._gemm_waves(a, w, out[:, :n], n, tc.STORE_BF16, bn, act=1)
    assert _close(out[:, :n], want.clamp(min=0) ** 2, 8)
    f32 = torch.full((m, n), 7.0, device=DEV)
    assert tc._gemm_waves(a, w, f32, n, tc.STORE_F32, bn) and _close(f32, want, 17)
    assert tc._gemm_waves(a, w, f32, n, tc.ACCUM_F32, bn) and _close(f32, 2 * want, 17)
    tc.check_status(DEV)


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("m,inter,k", [(3, 64, 64), (130, 264, 72), (2100, 1288, 136)])
def test_gated_pairs_in_waves(m, inter, k, bn):
    from types import SimpleNamespace
    from crucible_b200.ops import tensor_core as tc
    a, w, p = _inputs(m, 2 * inter, k, m + k)
    out = torch.empty(m, inter, device=DEV, dtype=torch.bfloat16)
    # (tanh.approx: 2^-11 of a gate, beside the result's rounding)
    assert tc._gemm_waves(a, w, out, inter, tc.SWIGLU_BF16, bn) and _close(out, _gated(p), 7.5)
    limit, alpha, offset = 1.25, 1.7, 1.0
    assert tc._gemm_waves(a, w, out, inter, tc.SWIGLU_BF16, bn, pair=(limit, alpha, offset))
    g, u = p.chunk(2, 1)
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    assert _close(out, g * torch.sigmoid(alpha * g) * (u + offset), 7.5)
    parts, eps = 3, 1e-5                          # rows ahead of their norm
    sumsq = torch.rand(parts, m, device=DEV) * k / parts
    pre = SimpleNamespace(sumsq=sumsq, parts=parts, x=a, eps=eps)
    assert tc._gemm_waves(a, w, out, inter, tc.SWIGLU_BF16, bn, pre=pre)
    assert _close(out, _gated(p / torch.sqrt(sumsq.double().sum(0) / k + eps)[:, None]), 7.5)
    tc.check_status(DEV)


@pytest.mark.parametrize("rows", [[1, 0, 127, 128, 129, 3], [700, 0, 0, 1, 640, 300]])
@pytest.mark.parametrize("gated", [False, True])
def test_grouped_products_in_waves(rows, gated):
    from crucible_b200.ops import tensor_core as tc
    e, k, n = len(rows), 136, 776
    pairs, tiles = sum(rows), [(x, sum(rows[:x]) + i, min(128, r - i)) for x, r in enumerate(rows) for i in range(0, r, 128)]
    most = len(tiles) + 5                         # entries beyond those in use are garbage
    plan = torch.full((2 + e + 3 * most,), 1 << 20, dtype=torch.int32)
    plan[0] = len(tiles)
    for i, t in enumerate(tiles):
        for j in range(3):
            plan[2 + e + j * most + i] = t[j]
    g = torch.Generator().manual_seed(pairs)
    a = torch.randn(pairs, k, generator=g).to(DEV).bfloat16()
    w = (torch.randn(e, (2 if gated else 1) * n, k, generator=g) * k ** -0.5).to(DEV).bfloat16()
    args = tc._NormArgs()
    plan = plan.to(DEV)
    args.plan, args.n_experts, args.max_tiles, args.w_rows = plan.data_ptr(), e, most, w.shape[1]
    for dtype in ([torch.bfloat16] if gated else [torch.float32, torch.bfloat16]):
        out = torch.full((pairs, n), 7.0, device=DEV, dtype=dtype)
        epi = tc.SWIGLU_BF16 if gated else tc.STORE_F32 if dtype == torch.float32 else tc.STORE_BF16
        assert tc._gemm_waves(a, w, out, n, epi, 256, plan=args)
        at = 0
        for x, r in enumerate(rows):
            p = a[at:at + r].double() @ w[x].double().T
            assert r == 0 or _close(out[at:at + r], _gated(p) if gated else p, 7.5 if dtype == torch.bfloat16 else 17)
            at += r
    tc.check_status(DEV)


def test_the_dispatch_reaches_it(monkeypatch):
    """Through the products' own entry points, at sizes on either side of the lines: which calls it ran, and that
    it refused none; the results against the kernel of a block a tile."""
    from types import SimpleNamespace
    from crucible_b200 import ops
    from crucible_b200.engine.context import Scratch
    from crucible_b200.ops import moe, tensor_core as tc
    calls, own = [], tc._gemm_waves
    monkeypatch.setattr(tc, "_gemm_waves", lambda *a, **kw: calls.append(own(*a, **kw)) or calls[-1])
    ctx = SimpleNamespace(scratch=Scratch(DEV).get)
    for m, n, k, kind, there in ((2050, 776, 136, "bf16", False), (1100, 8192, 64, "bf16", True), (1300, 4096, 128, "f32", True),
                                 (1100, 4096, 128, "f32", False), (300, 512, 64, "pair", False), (1664, 2048, 72, "pair", True)):
        a, w, want = _inputs(m, n * (2 if kind == "pair" else 1), k, m)
        ops.declare_weights(w)
        out = torch.full((m, n), 7.0, device=DEV, dtype=torch.float32 if kind == "f32" else torch.bfloat16)
        calls.clear()
        if kind == "pair":
            ops.linear_swiglu(a, w, out, ctx)
        else:
            ops.linear(a, w, out)
        assert calls == [True] * there, (m, n, k, kind)
        assert _close(out, _gated(want) if kind == "pair" else want, 17 if kind == "f32" else 7.5)
    experts, k, n = 2, 64, 1024
    for each, there in ((3200, True), (256, False)):
        tiles = experts * -(-each // 128)
        plan = torch.zeros(2 + experts + 3 * tiles, dtype=torch.int32)
        plan[0] = tiles
        for i in range(tiles):
            e, r = divmod(i * 128, -(-each // 128) * 128)
            for j, v in enumerate((e, e * each + r, min(128, each - r))):
                plan[2 + experts + j * tiles + i] = v
        a, w, _ = _inputs(experts * each, experts * n, k, each)
        w = w.view(experts, n, k)
        out = torch.full((experts * each, n), 7.0, device=DEV)
        calls.clear()
        assert moe.grouped_linear(a, w, out, plan.to(DEV), experts, tiles, False)
        assert calls == [True] * there
        want = torch.cat([a[e * each:(e + 1) * each].double() @ w[e].double().T for e in range(experts)])
        assert _close(out, want, 17)
    tc.check_status(DEV)
