"""What the batch builder keeps for the fixed block of a graph belongs to that block alone."""

import pytest
import torch

from oxr_inference_b200.cache import CacheManager, make_cache_plan
from oxr_inference_b200.engine.batch import BatchBuilder, Layout, StepEntry
from oxr_inference_b200.parts.base import PagedKVNeed, StateNeed


def test_a_block_that_has_a_dropped_blocks_id(monkeypatch):
    """Graphs that are dropped and captured anew: the next block may have the last one's id(), other requests and another size."""
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)      # no GPU here
    plan = make_cache_plan([PagedKVNeed(2, 16, 0), StateNeed((4,))], [None, None])
    cache = CacheManager(plan, page_size=8, num_pages=16, max_requests=4, device=torch.device("cpu"), dtype=torch.float32)
    builder = BatchBuilder(cache, [(16, 1, 8)], torch.device("cpu"), torch.zeros(2, dtype=torch.int32))
    entries = []
    for i in range(3):
        request = cache.open(i)
        assert cache.reserve(request, 5)
        cache.advance(request, 4)
        entries.append(StepEntry(request, [7 + i], [0]))

    @torch.inference_mode()
    def block_of(requests):
        layout = Layout(requests, requests, requests, [4], builder.decode_tile_caps(requests))
        return layout, torch.full((layout.total,), -7, dtype=torch.int32)

    small, block = block_of(3)
    for _ in range(2):      # rows filled, and then moved on by what a token moves alone
        builder.build(entries, layout=small, device_block=block, copy=False)
    taken, others = id(block), []
    del block
    for _ in range(100):
        large, block = block_of(4)
        if id(block) == taken:
            break
        others.append(block)
    if id(block) != taken:
        pytest.skip("the allocator gave the id to nobody")
    ctx = builder.build([], layout=large, device_block=block, copy=False)
    staging = builder.staging_of(block)
    assert staging.numel() == large.total
    at, size = large.offsets["state_slots"]
    assert staging[at:at + size].tolist() == [cache.scratch_slot] * 4, "padding rows alone"
    for view in (ctx.token_ids, ctx.state_slots, ctx.groups[0].block_table):
        assert block.data_ptr() <= view.data_ptr() < block.data_ptr() + 4 * large.total, "the step would read the block that is gone"
    ctx = builder.build(entries, layout=large, device_block=block, copy=False)
    assert staging[at:at + size].tolist() == [e.cache.state_slot for e in entries] + [cache.scratch_slot]
