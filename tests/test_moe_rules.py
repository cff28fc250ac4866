"""Which steps of few tokens run their experts as grouped products: both sides of the lines."""
import pytest
import torch


@pytest.mark.parametrize("width,ff,experts,top,shared,tokens", [
    # (the least tokens that go by grouped products)
    (2048, 2816, 8, 1, 2816, 2), (2048, 2816, 8, 2, 2816, 2), (2048, 2816, 8, 3, 2816, 1), (2048, 2816, 16, 4, 0, 1),
    (2048, 2816, 16, 1, 0, 4), (2048, 1408, 64, 8, 0, 1), (2048, 1408, 64, 2, 0, 4), (2048, 1408, 64, 2, 2816, 2),
    (4096, 1536, 128, 8, 0, 2), (1024, 1408, 32, 6, 0, 2), (1024, 1408, 32, 8, 0, 1), (1024, 1408, 8, 1, 1408, 3),
    (2048, 768, 128, 8, 0, 2), (2048, 768, 128, 4, 0, 4), (1024, 512, 64, 6, 1024, 2), (1024, 512, 64, 4, 0, 4)])
def test_where_experts_run_as_grouped_products(width, ff, experts, top, shared, tokens):
    from crucible_b200.config.model_config import FeedForwardSpec
    from crucible_b200.parts import FEED_FORWARDS
    options = (("experts", experts), ("top", top)) + ((("shared_intermediate", shared),) if shared else ())
    part = FEED_FORWARDS.build("moe", FeedForwardSpec("moe", width, ff, options))
    part.dtype = torch.bfloat16
    assert part._grouped(tokens) and (tokens == 1 or not part._grouped(tokens - 1))
    part.dtype = torch.float32
    assert not part._grouped(64)
