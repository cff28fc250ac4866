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


@pytest.mark.parametrize("width,ff,shared,experts,top,tokens,rides", [
    (2048, 2816, 2816, 8, 2, 128, True), (1024, 1408, 2816, 8, 2, 128, True), (1024, 1408, 2816, 8, 2, 129, False),
    (1024, 1408, 0, 8, 2, 64, False),
    # (of one slice beyond 128 rows: layers measured to be quicker so by 2 to 18 %, or slower by 2 to 13 %)
    (2048, 2816, 2816, 8, 2, 136, False), (1024, 1408, 1408, 8, 2, 1706, True), (2048, 2816, 2816, 8, 2, 384, True), (2048, 2816, 2816, 8, 2, 600, True),
    (2048, 2816, 2816, 8, 2, 1600, False), (2048, 2816, 2816, 8, 2, 2048, True), (2048, 2816, 2816, 8, 2, 4096, False),
    (1024, 1408, 1408, 8, 2, 136, True), (1024, 1408, 1408, 8, 2, 600, True), (2048, 1408, 1408, 32, 4, 450, True),
    (2048, 1408, 1408, 32, 4, 900, False), (1024, 1024, 1024, 16, 2, 256, True), (1024, 1024, 1024, 16, 2, 512, False),
    (4096, 1536, 1536, 8, 1, 384, False), (4096, 1536, 1536, 8, 1, 2048, True), (2048, 768, 768, 32, 8, 320, True),
    (2048, 768, 768, 32, 8, 2300, False), (3072, 2048, 2048, 8, 3, 230, False), (1024, 2816, 2816, 4, 1, 1000, True),
    (1024, 2816, 2816, 4, 1, 8192, False)])
def test_where_a_plain_shared_expert_rides(width, ff, shared, experts, top, tokens, rides):
    from crucible_b200.config.model_config import FeedForwardSpec
    from crucible_b200.parts import FEED_FORWARDS
    options = (("experts", experts), ("top", top)) + ((("shared_intermediate", shared),) if shared else ())
    part = FEED_FORWARDS.build("moe", FeedForwardSpec("moe", width, ff, options))
    part.dtype = torch.bfloat16
    assert part._rides(tokens) == rides


@pytest.mark.parametrize("pairs,experts", [(100, 64), (900, 8), (4096, 8), (24576, 64), (7, 3), (1, 256)])
def test_tiles_that_chance_fills(pairs, experts):
    """Against 400 draws; their mean is off by 4 of its own deviations at most, and the normal law by a tile in a hundred."""
    from crucible_b200.ops import tensor_core
    g = torch.Generator().manual_seed(pairs)
    drawn = torch.randint(experts, (400, pairs), generator=g)
    tiles = torch.stack([-(-torch.bincount(d, minlength=experts) // 128) for d in drawn]).sum(1).double()
    near = 4 * float(tiles.std()) / 20 + 0.01 * experts
    if pairs >= 30 * experts:                          # (fewer rows are no normal law; what matters then is below one tile each)
        assert abs(tensor_core.tiles_by_chance(pairs, experts) - float(tiles.mean())) <= near
    assert 0 < tensor_core.tiles_by_chance(pairs, experts) <= pairs / 128 + experts
