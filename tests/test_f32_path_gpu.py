"""The kernels of the 32-bit path alone: attention over tiles of keys and the CUDA-core product, against
float64, and the same bits for a row whatever runs beside it."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _attend(portions, firsts, q, gate, sinks, cache, table, H, G, D, E, window, keep, chunked, per_head):
    """Rows of several requests (tokens portions[r] at positions firsts[r] ...) through the wrapper."""
    from crucible_b200.ops import sink_attention
    starts, rows, req = [0], [], []
    for r, (n, f) in enumerate(zip(portions, firsts)):
        starts.append(starts[-1] + n)
        rows += list(range(f, f + n))
        req += [r] * n
    ctx = SimpleNamespace(n_requests=len(portions), req_row_start=_i32(starts), req_first_pos=_i32(firsts),
                          positions=_i32(rows), row_request=_i32(req), block_table=lambda g: table,
                          host=SimpleNamespace(max_new_tokens=max(portions)))
    out = torch.full((q.shape[0], H * E), float("nan"), device=DEV)
    sink_attention.attention(q, gate, out, sinks, H, G, D, E, D ** -0.5, window, keep, 0.7, ctx, cache,
                             SimpleNamespace(slot=0, group=0), gate_per_head=per_head, chunked=chunked)
    return out


@pytest.mark.parametrize("H,G,D,E,page,window,keep,chunked,per_head,sink", [
    (6, 2, 64, 64, 16, None, 0, False, False, True), (4, 1, 20, 36, 8, 70, 5, False, False, False),
    (4, 4, 128, 100, 32, 64, 0, True, True, True), (3, 1, 256, 256, 16, None, 0, False, False, False),
    (2, 1, 144, 132, 3, 33, 40, False, True, True)])
def test_attention_rows_have_their_own_bits(H, G, D, E, page, window, keep, chunked, per_head, sink):
    from crucible_b200 import ops
    g = torch.Generator().manual_seed(D)
    lengths = [197, 64]
    per = -(-max(lengths) // page)
    table = torch.randperm(2 * per, generator=g).to(torch.int32).view(2, per).to(DEV)
    k, v = (torch.randn(2 * per, G, page, n, generator=g).to(DEV) for n in (D, E))
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    q = [torch.randn(n, H * D, generator=g) for n in lengths]
    gate = [torch.randn(n, H if per_head else H * E, generator=g) for n in lengths]
    sinks = torch.randn(H, generator=g)
    on = lambda x: x.to(DEV).contiguous()
    args = (on(sinks) if sink else None, cache)
    opts = (H, G, D, E, window, keep, chunked, per_head)
    before = ops.LAUNCHES[0]
    whole = _attend(lengths, [0, 0], on(torch.cat(q)), on(torch.cat(gate)), *args, table, *opts)
    assert ops.LAUNCHES[0] == before + 1
    whole = [whole[:lengths[0]], whole[lengths[0]:]]
    for r, n in enumerate(lengths):
        pos = torch.arange(n)
        place = table[r].cpu().long()[pos // page]
        kk = k.cpu().double()[place, :, pos % page].repeat_interleave(H // G, 1)       # [n, H, D]
        vv = v.cpu().double()[place, :, pos % page].repeat_interleave(H // G, 1)
        s = torch.einsum("ihd,jhd->hij", q[r].double().view(n, H, D), kk) * D ** -0.5
        i, j = pos[:, None], pos[None]
        seen = j <= i
        if window:
            near = (i // window == j // window) if chunked else (i - j < window)
            seen = seen & (near | (j < keep))
        s = s.masked_fill(~seen, float("-inf"))
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(H, n, 1)], -1)
        want = torch.einsum("hij,jhe->ihe", torch.softmax(s, -1)[..., :n], vv)
        gt = torch.sigmoid(gate[r].double())
        want = want * (gt[:, :, None] if per_head else gt.view(n, H, E)) * 0.7
        err = float((whole[r].cpu().double().view(n, H, E) - want).abs().max() / want.abs().max())
        assert err < 2e-6, (r, err)                # float32 sums of at most 256 products and 197 keys
    # portions, single tokens (the form of few rows) and another request beside them: the same bits
    for cuts in ([100, 97], [1] * 3 + [194], [196, 1]):
        at = 0
        for n in cuts:
            portions, firsts = ([n, 64], [at, 0]) if n > 1 else ([n], [at])
            qq = torch.cat([q[0][at:at + n]] + ([q[1]] if n > 1 else []))
            gg = torch.cat([gate[0][at:at + n]] + ([gate[1]] if n > 1 else []))
            got = _attend(portions, firsts, on(qq), on(gg), *args, table, *opts)
            assert torch.equal(got[:n], whole[0][at:at + n]), (cuts, at)
            at += n
    # a later token's value that is not a number does not reach an earlier row
    v[table[0].long()[150 // page], :, 150 % page] = float("nan")
    again = _attend(lengths, [0, 0], on(torch.cat(q)), on(torch.cat(gate)), *args, table, *opts)
    assert torch.equal(again[:150], whole[0][:150]) and torch.equal(again[lengths[0]:], whole[1])
    assert bool(torch.isnan(again[150]).any())


@pytest.mark.parametrize("H,G,D,page,window,keep,chunked", [
    (4, 2, 64, 16, 70, 5, False), (2, 1, 144, 3, 33, 40, False), (4, 4, 128, 8, 64, 0, True)])
def test_pages_that_no_row_sees_are_not_read(H, G, D, page, window, keep, chunked):
    """Pages given back early (-1 in the table) lie in the tiles around a window and behind the kept tokens."""
    g = torch.Generator().manual_seed(page)
    firsts, portions = [360, 149], [41, 1]
    per = -(-(360 + 41) // page)
    table = torch.arange(2 * per, dtype=torch.int32).view(2, per)
    k, v = (torch.randn(2 * per, G, page, D, generator=g).to(DEV) for _ in range(2))
    cache = SimpleNamespace(keys=lambda s: k, values=lambda s: v, page_tokens=page)
    q, gate = (torch.randn(sum(portions), H * D, generator=g).to(DEV) for _ in range(2))
    opts = (None, cache)
    given_back = table.clone()
    for r, (first, n) in enumerate(zip(firsts, portions)):
        seen = torch.zeros(per * page, dtype=torch.bool)
        for pos in range(first, first + n):
            low = pos - pos % window if chunked else max(0, pos - window + 1)
            seen[low:pos + 1] = True
            seen[:min(keep, pos + 1)] = True
        given_back[r, ~seen.view(per, page).any(1)] = -1
    assert int((given_back < 0).sum()) > per
    outs = [_attend(portions, firsts, q, gate, *opts, t.to(DEV), H, G, D, D, window, keep, chunked, False)
            for t in (table, given_back)]
    assert torch.equal(*outs) and bool(torch.isfinite(outs[0]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 33, 20), (16, 64, 768), (17, 31, 19), (64, 65, 16), (130, 100, 1), (200, 77, 67)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_products_on_cuda_cores(dtype, M, N, K, accumulate):
    from crucible_b200.ops import build
    import ctypes
    lib = build.load("gemm_simt")
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).to(dtype).to(DEV), torch.randn(N, K, generator=g).to(dtype).to(DEV)
    c0 = torch.randn(M, N, generator=g).to(DEV)

    def product(rows):
        c = c0[:rows.shape[0]].clone()
        code = lib.cb_gemm_simt(*(ctypes.c_void_p(t.data_ptr()) for t in (rows, w, c)), 0 if dtype == torch.float32 else 1, 0,
                                rows.shape[0], N, K, K, K, N, int(accumulate), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert code == 0
        return c
    got = product(a)
    # the definition: one sum over k in ascending order, a multiply-add a step
    want = torch.zeros(M, N, dtype=torch.float64)
    for k in range(K):
        step = a[:, k].cpu().double()[:, None] * w[:, k].cpu().double()[None]
        want = (want + step).float().double()     # (a product of float32 numbers is exact in float64)
    want = want.float()
    if accumulate:
        want = c0.cpu() + want
    assert torch.equal(got.cpu(), want)
    few = product(a[:min(M, 5)].contiguous())
    assert torch.equal(few[:1], got[:1])


@pytest.mark.parametrize("M,N,K", [(8, 4608, 64), (33, 2304, 36), (65, 1280, 128), (300, 1280, 68), (513, 768, 16)])
def test_products_of_every_form_are_one_ascending_sum(M, N, K):
    """Sizes of each of the four forms of the fp32 product, at the edges of their tiles and of a stage of K."""
    from crucible_b200 import ops
    g = torch.Generator().manual_seed(M * N + K)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    want = torch.zeros(M, N, dtype=torch.float64)
    for k in range(K):                            # (a product of float32 numbers is exact in float64)
        want = (want + a[:, k].double()[:, None] * w[:, k].double()[None]).float().double()
    got = torch.full((M, N + 4), 7.0, device=DEV)
    ops.linear_plain(a.to(DEV), w.to(DEV), got[:, :N])
    assert torch.equal(got[:, :N].cpu(), want.float()) and bool((got[:, N:] == 7.0).all())


@pytest.mark.parametrize("rows", [1, 40, 130])
@pytest.mark.parametrize("n,k,a_head,shift", [(192, 128, 192, 0), (33, 20, 24, 0), (64, 30, 31, 1)])
def test_products_per_head_are_the_products(rows, n, k, a_head, shift):
    from crucible_b200 import ops
    heads = 5
    g = torch.Generator().manual_seed(rows + n)
    a = torch.randn(rows, heads * a_head + shift, generator=g).to(DEV)[:, shift:]
    w = torch.randn(heads, n, k, generator=g).to(DEV)
    got = torch.zeros(rows, heads * n, device=DEV)
    want = got.clone()
    ops.linear_heads_plain(a, a_head, w, got, n)
    for h in range(heads):
        ops.linear_plain(a[:, h * a_head:h * a_head + k].contiguous(), w[h], want[:, h * n:h * n + n])
    assert torch.equal(got, want)
    with pytest.raises(ops.KernelError):
        ops.linear_heads_plain(a[:, :heads * a_head - a_head + k - 1], a_head, w, got, n)


@pytest.mark.parametrize("M,N,K", [(5, 1280, 16), (520, 1284, 136), (1300, 2050, 36), (700, 772, 36), (300, 2050, 20)])
def test_short_products_are_one_ascending_sum(M, N, K):
    """Sizes that go by the kernel whose stages are of 16, or by the forms beside its line."""
    from crucible_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    want = torch.zeros(M, N, dtype=torch.float64)
    for k in range(K):                            # (a product of float32 numbers is exact in float64)
        want = (want + a[:, k].double()[:, None] * w[:, k].double()[None]).float().double()
    got = torch.full((M, N + 4), 7.0, device=DEV)
    ops.linear_plain(a.to(DEV), w.to(DEV), got[:, :N])
    assert torch.equal(got[:, :N].cpu(), want.float()) and bool((got[:, N:] == 7.0).all())


def test_more_rows_than_tiles_of_sixteen_in_a_grid():
    from crucible_b200 import ops
    M, N, K = 16 * 65535 + 40, 8, 20
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    got = torch.full((M, N), 7.0, device=DEV)
    ops.linear_plain(a, w, got)
    few = torch.empty(37, N, device=DEV)
    ops.linear_plain(a[-37:], w, few)
    assert torch.equal(got[-37:], few)
    assert float((got.double() - a.double() @ w.double().T).norm() / got.double().norm()) < 1e-6      # (20 roundings of 2^-24)
