"""A whole slice scattered in one call (entries laid out by linear index, then
looked up by the inverse permutation) against the same blocks in two calls
(entry by entry, by the permutation): the same bytes, for sizes below and
above 2^32 entries, few and more shards than entries, part of the shards, both
address forms, and an odd address.  A batch that lacks a block, or has one
twice in place of another, is not a whole slice."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slice_,shards,lo,hi,own", [
    (0, 1, 0, 1, False), (0, 8, 0, 8, False), (1, 4, 1, 4, True), (3, 1, 0, 1, False), (3, 65536, 0, 65536, False),
    (3, 1 << 18, 1000, 200000, False), (4, 16, 5, 6, True), (5, 1024, 700, 1024, False), (6, 64, 0, 64, True),
    (10, 4096, 4000, 4002, False)])
def test_whole_slice_equals_its_halves(cuda, slice_, shards, lo, hi, own):
    import torch
    from pentago_b200 import capi, shard, supertensor
    m, blocks, nodes = shard.synthetic_slice(slice_, 3)
    loc = shard.shard_locator_t(shards)
    if own:   # shards in reverse order, a byte apart
        sizes = [loc.shard_size(m.total(), s) for s in range(lo, hi)]
        offsets = np.zeros(hi - lo, np.int64)
        at = 0
        for k in reversed(range(hi - lo)):
            offsets[k] = at
            at += sizes[k] + 1
        n = at
    else:
        offsets, q, r = None, m.total() // shards, m.total() % shards
        n = (hi - lo) * q + min(hi, r) - min(lo, r)

    def scatter(picks, turn):
        buf = torch.full((n + 8,), 9, dtype=torch.uint8, device="cuda")
        for pick in picks:
            part = (capi.pg_shard_block_t * len(pick))(*[blocks[i] for i in pick])
            capi.check(capi.lib().pg_shard_scatter(
                slice_, shards, lo, hi, part, len(part), nodes.data_ptr(), turn, buf.data_ptr() + 1,
                offsets.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)) if own else None, capi.stream_handle()))
        torch.cuda.synchronize()
        return buf

    every = list(range(len(blocks)))
    half = len(every) // 2
    for turn in (supertensor.RAW, 0, 1):
        whole = scatter([every], turn)
        if half:
            assert torch.equal(whole, scatter([every[:half], every[half:]], turn))
        assert whole[0] == 9 and (whole[n + 1:] == 9).all()
        if slice_ > 9:
            return
    if half:
        # the last block missing, or the first in its place
        lacking = scatter([every[:-1]], 0)
        assert torch.equal(lacking, scatter([every[:half], every[half:-1]], 0))
        same = [i for i in every[:-1] if bytes(blocks[i])[:4] == bytes(blocks[every[-1]])[:4]]
        assert torch.equal(scatter([every[:-1] + same[:1]], 0), lacking)
