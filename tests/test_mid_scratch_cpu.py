"""The scratch that a midsolve batch asks for: a board whose workspace lies in
shared memory needs a descriptor, a larger one its tables and workspace."""
import numpy as np

from pentago_b200 import mid


def boards(stones, n):
    return mid.random_boards(stones, n, stones)


def test_scratch_is_what_the_kernels_use():
    for stones in (26, 30, 36):
        assert 0 < mid.scratch_bytes(boards(stones, 64)) <= 64 * 64
    small, large = boards(28, 5), boards(21, 3)
    alone, both = mid.scratch_bytes(large), mid.scratch_bytes(np.concatenate([small, large]))
    assert alone >= 3 * 16 * mid.workspace_size(21)       # halfsupers of 16 bytes
    assert alone < both <= alone + 5 * 64 + 256           # (descriptors lie on 256-byte boundaries)
