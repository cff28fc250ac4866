"""Which single tokens go by one block a request and key/value head: both sides of the lines of
`short_attention_pays`, and the class of short contexts that a step's key tells apart."""
import pytest


@pytest.mark.parametrize("blocks,reach,head_dim,plain,group,pays", [
    # against the tcgen05 kernel: one tile of keys has nothing to merge
    (4, 128, 64, True, 3, False), (4, 256, 64, True, 3, True), (4, 128, 128, True, 4, True), (4, 128, 128, True, 8, False),
    (4, 256, 128, True, 8, True), (148, 256, 64, True, 4, True), (149, 256, 64, True, 4, False),
    (4, 512, 64, True, 4, True), (16, 512, 64, True, 8, False), (24, 512, 64, True, 8, True), (4, 768, 64, True, 4, False),
    (32, 512, 128, True, 4, False), (48, 512, 128, True, 4, True), (192, 768, 128, True, 4, True), (96, 1024, 128, True, 4, True),
    (192, 1024, 128, True, 4, False), (48, 512, 128, True, 8, False), (96, 1280, 128, True, 4, False),
    # with a sink or a gate, against the mma.sync kernel
    (1, 1024, 64, False, 4, True), (1, 1024, 128, False, 1, True), (24, 1536, 64, False, 4, False), (32, 1536, 64, False, 4, True),
    (32, 2048, 128, False, 4, False), (48, 2048, 128, False, 4, True), (64, 3840, 64, False, 4, True), (64, 3840, 128, False, 4, False),
    (64, 8192, 64, False, 4, False), (96, 8192, 128, False, 4, True), (1000, 8448, 128, False, 4, False),
    (1, 512, 64, False, 8, True), (16, 768, 64, False, 8, False), (1, 256, 128, False, 8, True), (16, 512, 128, False, 8, False),
    (32, 512, 128, False, 8, True), (48, 1024, 128, False, 8, False), (96, 1536, 128, False, 8, True), (96, 2048, 128, False, 8, False)])
def test_where_one_block_walks_the_keys(blocks, reach, head_dim, plain, group, pays):
    from crucible_b200.ops import tensor_core as tc
    assert tc.short_attention_pays(blocks, reach, head_dim, plain, group) is pays


def test_short_contexts_of_many_tokens():
    from crucible_b200.ops import tensor_core as tc
    for tokens, pays in ((1, False), (16, False), (17, True), (37, True), (38, False)):
        assert tc.short_attention_pays(4 * tokens, 128, 64, True, 3, tokens) is pays
        assert tc.short_attention_pays(4 * tokens, 256, 64, True, 3, tokens) is (4 * tokens <= 148)


def test_one_long_context_among_short_ones_is_split():
    """16 users of 4 key/value heads, one behind 8,000 keys: the rule sees the longest."""
    from crucible_b200.engine.context import HostStep
    from crucible_b200.ops import tensor_core as tc
    host = HostStep(list(range(16)), [1] * 16, [8000] + [200] * 15, [8001] + [201] * 15, list(range(16)))
    for head_dim in (64, 128):
        for plain in (True, False):
            assert not tc.short_attention_pays(16 * 4, host.context_reach, head_dim, plain, 4)


def test_a_steps_key_tells_short_contexts_apart():
    from crucible_b200.engine.context import HostStep
    def step(new, held):
        after = [a + b for a, b in zip(new, held)]
        return HostStep(list(range(len(new))), new, held, after, list(range(len(new))))
    for longest, reach in ((1, 128), (128, 128), (129, 256), (256, 256), (257, 512), (2101, 2304)):
        one = step([1, 1], [longest - 1, 0])
        assert one.context_reach == one.lead_context_reach == reach
        assert one.context_bucket == one.lead_context_bucket == 256 * -(-longest // 256)
        assert one.shape_key() == (1, 2, reach, reach)
    mixed = step([1, 1, 500], [100, 127, 0])
    assert mixed.lead_context_reach == 128 and mixed.context_reach == 512 and mixed.shape_key() == (500, 2, 0, 128)
    assert step([1, 1, 500], [100, 128, 0]).shape_key() == (500, 2, 0, 256)
    prompts = step([70], [0])
    assert prompts.lead_context_reach == 0 and prompts.shape_key() == (70, 0, 0, 0)


@pytest.mark.parametrize("pages,heads,page,taken", [
    (64, 4, 16, True), ((1 << 31) // 64 - 1, 4, 16, True), ((1 << 31) // 64, 4, 16, False), (1 << 25, 16, 32, False)])
def test_32_bit_tiles_take_pools_whose_rows_an_int_counts(pages, heads, page, taken, monkeypatch):
    """Where a key lies is kept as an int, the row of the pool; a pool with more rows than that (heads of 4: from 34 GB on)
    goes by the kernels that reckon in 64 bits."""
    from types import SimpleNamespace
    import torch
    from crucible_b200 import ops
    calls = []
    monkeypatch.setattr(ops.build, "load", lambda name: SimpleNamespace(cb_attention_f32=lambda *a: calls.append(a) or 0))
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_ptr", lambda t: 0)
    pool = torch.zeros(4).expand(pages, heads, page, 4)              # (its size alone is real)
    rows, numbers = torch.zeros(3, 4 * heads), torch.zeros(4, dtype=torch.int32)
    ctx = SimpleNamespace(host=SimpleNamespace(max_new_tokens=3), req_row_start=numbers, req_first_pos=numbers, n_requests=1)
    got = ops.attention_f32(rows, None, torch.zeros(3, 4 * heads), pool, pool, None, heads, heads, 4, 4, 0.5, None, False, 0, 1.0,
                            ctx, page, torch.zeros((1, 4), dtype=torch.int32))
    assert got == taken and len(calls) == taken


@pytest.mark.parametrize("blocks,new,context,warps", [
    # (measured: 8 and 4 warps, us: 48 and 49, 90 and 97, 61 and 65; 202 and 197, 368 and 257, 179 and 160; 78 and 71)
    (172, 450, 450, 8), (176, 700, 700, 8), (197, 700, 700, 8), (136, 130, 1630, 8), (163, 130, 1630, 4), (195, 130, 1630, 4),
    (264, 700, 700, 4), (148, 90, 690, 8), (149, 90, 180, 4), (200, 90, 179, 8), (201, 90, 90, 4)])
def test_warps_of_a_32_bit_attention_block(blocks, new, context, warps):
    from crucible_b200 import ops
    assert ops.f32_attention_warps(blocks, new, context) == warps
