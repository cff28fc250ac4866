"""The walk over tokens with one, two and four columns of a matrix a lane: the same sums in the same order, so the
same bits, in results and states."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("rule", ["DELTA", "MLSTM", "WKV", "SSD", "CHANNEL"])
@pytest.mark.parametrize("H,G,D,E", [(4, 2, 128, 128), (3, 3, 100, 36), (2, 1, 64, 68), (2, 2, 40, 16), (2, 2, 64, 30), (2, 2, 16, 20)])
@pytest.mark.parametrize("lengths", [[1, 1, 1], [17], [5, 40, 1, 16]])
def test_columns_a_lane_change_no_bit(rule, H, G, D, E, lengths, monkeypatch):
    from crucible_b200.ops import recurrent as k
    code, T, R = getattr(k, rule), sum(lengths), len(lengths)
    g = torch.Generator().manual_seed(D + E)
    vector = rule in ("WKV", "CHANNEL")
    if vector and G != H:
        G = H
    C = 2 * G * D + H * E + (H * D if vector else 0)
    qkv = torch.randn(T, C, generator=g) * 0.3
    if vector:
        qkv[:, 2 * G * D + H * E:] = torch.rand(T, H * D, generator=g)
    sc0, sc1 = torch.rand(T, H, generator=g), torch.rand(T, H, generator=g)
    nbytes = -(-4 * (H * D * E + H * D + H) // 16) * 16
    before = torch.randn(R, nbytes // 4, generator=g) * 0.3
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=_i32(starts), req_state_slot=_i32(list(range(R))),
                          dtype=torch.float32, host=None, scratch=None)
    per = torch.randn(H, D, generator=g) if rule == "WKV" else torch.randn(H, generator=g) if rule == "SSD" else None
    q, s0, s1, p = (t.to(DEV) if t is not None else None for t in (qkv, sc0, sc1, per))
    kept = (torch.randn(R, H * (D + 1), generator=g) * 0.3).to(DEV) if rule == "MLSTM" else None
    got = {}
    for columns in (1, 2, 4):
        monkeypatch.setattr(k, "walk_columns", lambda *a: (columns, 0.0))
        state = before.clone().to(DEV).view(torch.uint8)
        out = torch.full((T, H * E), float("nan"), device=DEV)
        k.matrix_memory(code, q, 0, G * D, 2 * G * D, s0, s1, ctx, state, 0, 4 * H * D * E, 4 * (H * D * E + H * D), out,
                        H, G, D, E, w_off=2 * G * D + H * E, per_head=p, kept=kept)
        got[columns] = out, state
    assert not torch.isnan(got[1][0]).any()
    for columns in (2, 4):
        assert torch.equal(got[columns][0], got[1][0]) and torch.equal(got[columns][1], got[1][1])
