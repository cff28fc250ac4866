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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shared,slices,copies", [(0, 0, 1), (64, 1, 1), (60, 1, 1), (100, 0, 1), (124, 2, 1), (120, 2, 2)])
def test_a_shared_expert_is_held_once(shared, slices, copies, dtype):
    """One whose slice rides with the routed experts has no second copy for the steps in which it does not; one of several
    slices has, unless it is of a size that the dense products refuse."""
    from crucible_b200.config.model_config import FeedForwardSpec
    from crucible_b200.parts import FEED_FORWARDS
    width, ff, experts = 32, 64, 4
    options = (("experts", experts), ("top", 2)) + ((("shared_intermediate", shared),) if shared else ())
    part = FEED_FORWARDS.build("moe", FeedForwardSpec("moe", width, ff, options))
    given = {t.name: torch.randn(t.shape).to(dtype) for t in part.tensors()}
    part.bind(given, dtype, torch.device("cpu"))
    held, todo = {}, [part]
    while todo:
        x = todo.pop()
        if isinstance(x, torch.Tensor):
            held[x.untyped_storage().data_ptr()] = x.untyped_storage().nbytes()
        elif isinstance(x, (list, tuple)):
            todo += x
        elif x is part or (x is not None and x is part.shared):
            todo += vars(x).values()
    size = torch.finfo(dtype).bits // 8
    matrices = sum(t.numel() for n, t in given.items() if n != "router")
    assert part.slices == (slices if dtype == torch.bfloat16 else 0)
    more = 3 * width * (part.slices * ff - shared if part.slices and copies == 1 else part.slices * ff)
    assert sum(held.values()) == (matrices + more + given["router"].numel()) * size + 4 * (experts + part.slices)


@pytest.mark.parametrize("width,ff,shared,tokens,rides", [
    (2048, 2816, 2816, 128, True), (2048, 2816, 2816, 129, False), (2048, 2816, 2816, 319, False), (2048, 2816, 2816, 320, True),
    (2048, 2816, 2816, 2048, True), (2048, 2816, 2816, 2049, False), (1024, 1408, 1408, 129, True), (1024, 1408, 1408, 2048, True),
    (1024, 1408, 2816, 128, True), (1024, 1408, 2816, 129, False), (1024, 1408, 0, 64, False)])
def test_where_a_plain_shared_expert_rides(width, ff, shared, tokens, rides):
    from crucible_b200.config.model_config import FeedForwardSpec
    from crucible_b200.parts import FEED_FORWARDS
    options = (("experts", 8), ("top", 2)) + ((("shared_intermediate", shared),) if shared else ())
    part = FEED_FORWARDS.build("moe", FeedForwardSpec("moe", width, ff, options))
    part.dtype = torch.bfloat16
    assert part._rides(tokens) == rides
