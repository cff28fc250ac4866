"""The rotation's tables: cosine and sine of position times frequency, every entry the float32 nearest to them."""
import math

import pytest
import torch


@pytest.mark.parametrize("theta,dim,positions", [(10000.0, 64, 4096), (500000.0, 128, 700), (1e6, 2, 33)])
def test_every_entry_is_the_nearest_float32(theta, dim, positions):
    from crucible_b200.config.model_config import PositionSpec
    from crucible_b200.parts import POSITIONS
    rope = POSITIONS.build("rope", PositionSpec("rope", dim, theta, positions))
    rope.bind({}, torch.float32, torch.device("cpu"))
    for table, f in ((rope.cos, math.cos), (rope.sin, math.sin)):
        assert table.shape == (positions, dim // 2) and table.dtype == torch.float32 and table.is_contiguous()
        want = torch.tensor([[f(p * theta ** (-2.0 * i / dim)) for i in range(dim // 2)] for p in range(positions)],
                            dtype=torch.float64)
        near = want.to(torch.float32)
        # (the frequency's last bit of 64 times the position may move an entry that lies between two float32 numbers)
        off = table != near
        assert int(off.sum()) <= 2e-6 * off.numel() + 1
        assert float((table.double() - want).abs().max()) <= 2.0 ** -25 + positions * 2.0 ** -50
