"""Which form of the walk over tokens a step is given (no GPU: the entry points are stand-ins)."""
from types import SimpleNamespace

import pytest
import torch

STEPS = [([700, 123, 246], 8, 128), ([700, 123], 16, 128), ([300, 300], 16, 128), ([450] * 4, 8, 128), ([600, 410, 520], 16, 64),
         ([300, 700, 410, 520, 333], 8, 128), ([300, 700, 410, 520, 333], 16, 128), ([600] + [1] * 12, 16, 128),
         ([24] * 32, 16, 128), ([1] * 32, 8, 128)]


def _columns(rule, lengths, H, D, dtype, counts, monkeypatch):
    """What `matrix_memory` asks of the walk for portions of `lengths`."""
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import build, recurrent as k
    seen = []
    lib = SimpleNamespace(cb_matrix_memory=lambda *a: seen.append(a[-2]) or 0,
                          cb_matrix_memory_step=lambda *a: build.UNSUPPORTED)
    monkeypatch.setattr(k.build, "load", lambda name: lib)
    monkeypatch.setattr(k, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(k, "_stream", lambda: 0)
    monkeypatch.setattr(k, "CHUNKS", False)
    R, T = len(lengths), sum(lengths)
    vector = rule in (k.WKV, k.CHANNEL)
    numbers = torch.zeros(T, H)
    starts = torch.zeros(R + 1, dtype=torch.int32)
    held = [5] * R
    ctx = SimpleNamespace(n_requests=R, n_tokens=T, req_row_start=starts, req_state_slot=starts, dtype=dtype,
                          host=HostStep(list(range(R)), lengths, held, [5 + n for n in lengths], held) if counts else None)
    k.matrix_memory(rule, torch.zeros(T, 3 * H * D + H * D * vector), 0, H * D, 2 * H * D, numbers, numbers, ctx,
                    torch.zeros((R, 4 * (H * D * D + H * D + H)), dtype=torch.uint8), 0, 4 * H * D * D, 4 * H * D * (D + 1),
                    torch.empty(T, H * D), H, H, D, D, w_off=3 * H * D, kept=torch.zeros(R, H * (D + 1)))
    return seen


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rule", ["DELTA", "MLSTM", "WKV", "SSD", "CHANNEL"])
@pytest.mark.parametrize("lengths,H,D", STEPS)
def test_a_step_is_walked_in_the_form_its_lengths_ask_for(rule, lengths, H, D, dtype, monkeypatch):
    """In 32 bits (which always walk) as in 16: by the portions' number, tokens and longest."""
    from crucible_b200.ops import recurrent as k
    code = getattr(k, rule)
    got = _columns(code, lengths, H, D, dtype, True, monkeypatch)
    assert got == [k.walk_columns(code, len(lengths), sum(lengths), max(lengths), H, D, D)[0]]
    if len(lengths) * H * (D // 16) <= 148:
        assert got == [1]                              # up to a block an SM
    elif max(lengths) >= 300 and sum(lengths) < 2 * max(lengths) and rule in ("DELTA", "MLSTM", "CHANNEL"):
        assert got[0] < 4                              # (four take half as long again over a long portion)


@pytest.mark.parametrize("rule", ["DELTA", "MLSTM", "WKV", "SSD", "CHANNEL"])
def test_portions_of_unknown_length_have_a_column_a_lane(rule, monkeypatch):
    from crucible_b200.ops import recurrent as k
    for dtype in (torch.float32, torch.bfloat16):
        assert _columns(getattr(k, rule), [700, 123, 246], 8, 128, dtype, False, monkeypatch) == [1]


@pytest.mark.parametrize("rule,lengths,H,D,columns", [
    # (measured: the quickest of one, two and four)
    ("DELTA", [180, 1, 75, 40, 9, 130], 16, 128, 1), ("SSD", [180, 1, 75, 40, 9, 130], 16, 128, 1), ("DELTA", [900, 300, 300, 300], 32, 128, 1),
    ("WKV", [600] + [1] * 12, 16, 64, 1), ("WKV", [400, 1, 1, 1], 32, 128, 1), ("DELTA", [300, 700, 410, 520, 333], 16, 64, 1),
    ("DELTA", [300, 700, 410, 520, 333], 8, 128, 1), ("MLSTM", [330, 290], 32, 128, 2), ("DELTA", [450] * 4, 16, 128, 2),
    ("MLSTM", [450] * 4, 16, 128, 2), ("SSD", [24] * 32, 16, 128, 4)])
def test_more_columns_only_where_they_are_clearly_quicker(rule, lengths, H, D, columns):
    from crucible_b200.ops import recurrent as k
    assert k.walk_columns(getattr(k, rule), len(lengths), sum(lengths), max(lengths), H, D, D)[0] == columns


@pytest.mark.parametrize("rule,lengths,heads", [
    # (measured, chunks and walk, us: 239 and 342, 300 and 373, 222 and 316, 212 and 313, 268 and 352, 178 and 274, 41 and
    # 51, 64 and 87)
    ("DELTA", [300, 700, 410, 520, 333], 16), ("CHANNEL", [300, 700, 410, 520, 333], 16),
    ("DELTA", [500, 250, 125, 60, 30], 32), ("DELTA", [64, 128, 256, 512], 32), ("DELTA", [513, 511, 300], 32),
    ("CHANNEL", [330, 290], 32), ("SSD", [150, 100, 120], 16), ("SSD", [150, 100, 120], 32)])
def test_the_walk_that_chunks_are_weighed_against_is_the_one_launched(rule, lengths, heads):
    from crucible_b200.ops import recurrent as k
    code, shape = getattr(k, rule), (sum(lengths), len(lengths), max(lengths))
    assert k.chunks_pay(code, *shape, float(heads))
    first, chunk = k.COSTS[code][1]
    walk = k.walk_columns(code, len(lengths), sum(lengths), max(lengths), heads, 128, 128)[1]
    assert walk > first + chunk * (sum(lengths) / 32 + len(lengths) / 2) * heads
