"""The delta rules' walk over chunks where heads of 64 have more blocks than SMs, two to an SM: the bits that the same
portions have one at a time, a block an SM."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rule", ["DELTA", "CHANNEL"])
@pytest.mark.parametrize("H,G,D,E", [(28, 28, 64, 64), (28, 14, 64, 36), (30, 30, 40, 36)])
def test_portions_together_have_the_bits_of_each(rule, H, G, D, E, monkeypatch):
    from crucible_b200.ops import recurrent as k
    from crucible_b200.ops import tensor_core
    monkeypatch.setattr(k, "chunks_pay", lambda *a: True)
    code, lengths = getattr(k, rule), [33, 97, 5, 64]
    if rule == "CHANNEL":
        G = H
    g = torch.Generator().manual_seed(D + E)
    T, C = sum(lengths), 2 * G * D + H * E + (H * D if rule == "CHANNEL" else 0)
    qkv = torch.randn(T, C, generator=g) * 0.2
    if rule == "CHANNEL":
        qkv[:, 2 * G * D + H * E:] = torch.rand(T, H * D, generator=g) ** 0.1
    sc0, sc1 = torch.rand(T, H, generator=g) ** 0.1, torch.rand(T, H, generator=g)
    before = torch.randn(len(lengths), H * D * E, generator=g) * 0.3
    qkv, sc0, sc1 = (t.to(DEV) for t in (qkv, sc0, sc1))

    def walked(first, last, begin):
        lens = lengths[first:last]
        starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
        rows = slice(begin, begin + sum(lens))
        ctx = SimpleNamespace(dtype=torch.bfloat16, n_requests=len(lens), req_row_start=starts.to(DEV),
                              req_state_slot=torch.arange(len(lens), dtype=torch.int32, device=DEV),
                              scratch=lambda name, shape, kind: torch.full(tuple(shape), float("nan"), dtype=kind, device=DEV),
                              host=SimpleNamespace(max_new_tokens=max(lens), lead_single=0))
        state = before[first:last].clone().to(DEV)
        out = torch.full((sum(lens), H * E), float("nan"), device=DEV)
        k.matrix_memory(code, qkv[rows], 0, G * D, 2 * G * D, sc0[rows], sc1[rows], ctx, state.view(torch.uint8), 0, 0, 0, out,
                        H, G, D, E, w_off=2 * G * D + H * E)
        return out, state

    together, states = walked(0, len(lengths), 0)
    assert not torch.isnan(together).any()
    begin = 0
    for i, n in enumerate(lengths):
        alone, state = walked(i, i + 1, begin)
        assert torch.equal(together[begin:begin + n], alone) and torch.equal(states[i], state[0])
        begin += n
    tensor_core.check_status(DEV)
