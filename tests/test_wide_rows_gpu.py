"""Latent attention over cached rows of 256 features on the tcgen05 tiles: prompts and portions at the
edges of tiles of keys and of packed query rows, windows, a sink, scattered pages and pages that
follow one another, against the plain functions in float64 and against the mma.sync tiles."""
import pytest
import torch

import plain_nipapel
import plain_sebalorn
import test_nipapel_kernels_gpu as nipapel
import test_sebalorn_kernels_gpu as sebalorn
from test_futepel_kernels_gpu import TOL, _bind, _binding, rel
from test_nipapel_kernels_gpu import StepsWithValues, _run_part

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _counted(monkeypatch):
    from crucible_b200.ops import tensor_core
    seen, real = [], tensor_core._attention_tcgen05

    def spy(*a, **k):
        seen.append(real(*a, **k))
        return seen[-1]
    monkeypatch.setattr(tensor_core, "_attention_tcgen05", spy)
    return seen


def _in_order(steps):
    steps.tables = torch.arange(steps.tables.numel(), dtype=torch.int32).view(steps.tables.shape)


@pytest.mark.parametrize("H,C,R,page,window,cuts,ordered", [
    (16, 192, 64, 16, None, [300], False),       # 37 and a half tiles of rows, three tiles of keys
    (16, 192, 64, 16, None, [8, 120, 1, 7, 129], True),     # portions at and beside the edges of 128 keys
    (4, 192, 64, 128, 100, [250], True),         # a page a tile; a window inside a tile
    (3, 256, 0, 8, 200, [64, 300], False),       # nothing turned; groups that do not divide a tile of rows
    (1, 224, 32, 64, None, [64, 66], True)])     # one head: a row a token
def test_windows_and_edges(H, C, R, page, window, cuts, ordered, monkeypatch):
    from crucible_b200.ops import tensor_core
    from crucible_b200.parts import MIXERS
    width, T, D, E, Q = 64, sum(cuts), 16, 24, 40
    part = MIXERS.build("latent_attention", nipapel._latent_spec(H, D, R, E, C, Q, width, window))
    w = _bind(part, BF16, 9, std=0.2)
    h = {0: torch.randn(T, width).to(BF16).float()}
    seen, got = _counted(monkeypatch), []
    for use in (True, False):
        monkeypatch.setattr(tensor_core, "USE_TCGEN05_ATTENTION", use)
        steps = StepsWithValues(BF16, part.cache_need(), page, 1, 512, seed=4)
        if ordered:
            _in_order(steps)
        got.append(_run_part(part, steps, [[(0, n)] for n in cuts], h, width, _binding(part, group=0))[0])
    assert seen.count(True) == sum(n * H >= 64 for n in cuts)
    pos, x = torch.arange(T), h[0].double()
    if R:
        cfg = nipapel._latent_cfg(H, D, R, E, C, Q, window)
        ref = plain_nipapel.latent_attention(x, w, cfg, 1e-5, pos, plain_nipapel.latent_rows(x, w, cfg, 1e-5, pos))
        assert rel(got[0], ref) < TOL[BF16]
    # both forms round the same scores and probabilities to bfloat16, in another order
    assert rel(got[0], got[1]) < TOL[BF16]


@pytest.mark.parametrize("schedule", [[[(0, 200), (1, 33)]], [[(0, 70), (1, 33)], [(0, 130)]]])
def test_with_a_sink(schedule, monkeypatch):
    from crucible_b200.parts import MIXERS
    H, D, R, E, C, Q, width = 5, 16, 64, 16, 192, 24, 64
    scale = 2.5 / (0.09 * (C * Q * D) ** 0.5)
    part = MIXERS.build("latent_attention", sebalorn._latent_spec(H, D, R, E, C, Q, width, scale))

    def edit(t):
        t["sink"] = torch.linspace(6.0, -6.0, H)
    w = _bind(part, BF16, 9, std=0.3, edit=edit)
    h = {0: torch.randn(200, width).to(BF16).float(), 1: torch.randn(33, width).to(BF16).float()}
    seen = _counted(monkeypatch)
    steps = StepsWithValues(BF16, part.cache_need(), 16, 2, 256, seed=4)
    got = _run_part(part, steps, schedule, h, width, _binding(part, group=0))
    assert len(seen) == len(schedule) and all(seen)
    cfg = sebalorn._latent_cfg(H, D, R, E, C, Q, scale)
    for slot, x in h.items():
        assert rel(got[slot], plain_sebalorn.latent_attention(x.double(), w, cfg, 1e-5, "")) < TOL[BF16]


@pytest.mark.parametrize("D", [256, 80])
@pytest.mark.parametrize("chunks,requests,window", [
    (1, [(1, 255), (2, 3)], None),                # nothing to merge
    (2, [(1, 400), (1, 3)], None),                # rows of one chunk are written at once
    (9, [(1, 2100), (2, 250), (1, 0)], None),
    (33, [(1, 8200), (3, 8190)], None),           # one chunk beyond 32 at a time
    (33, [(1, 8200), (2, 8191)], 700)])           # a window: the row's own chunks alone
def test_decoded_rows_of_many_chunks(D, chunks, requests, window, monkeypatch):
    """A decoded row's keys in chunks, merged by a kernel of their own; heads that fill no tile."""
    from test_kernels_gpu import _paged_case
    from crucible_b200.ops import tensor_core
    keys = 64 if D > 128 else 256
    if D > 128:                                   # (chunks of 64 keys)
        requests = [(n, h // 4) for n, h in requests]
        window = window and window // 4
    H, G = 10, 2
    qkv, ctx, cache, binding, ref = _paged_case(BF16, H, G, D, 16, [(h, n) for n, h in requests], 7, window)
    monkeypatch.setattr(tensor_core, "wide_row_chunk_keys", lambda *a: keys)
    monkeypatch.setattr(tensor_core, "decode_chunk_keys", lambda *a: keys)
    longest = max(n + h for n, h in requests)
    assert -(-longest // keys) == chunks and ctx.host.max_new_tokens * (H // G) <= tensor_core.SPLIT_ROWS
    out = torch.full((qkv.shape[0], H * D), float("nan"), device="cuda:0", dtype=BF16)
    assert tensor_core.paged_attention(qkv, out, H, G, D, D ** -0.5, window, ctx, cache, binding)
    assert rel(out.cpu(), ref) < TOL[BF16]
