"""The midsolve index tables are checked before they go to a device: the pass
kernel reads and writes where they say, for any board, without looking."""
import numpy as np
import pytest

from pentago_b200 import capi

PG_ERR_BOUNDS = capi.PG_ERR_BOUNDS


def check(spots, what, at, delta):
    return capi.lib().pg_selftest_small_tables(spots, what, at, delta)


@pytest.mark.parametrize("spots", range(11))
def test_the_tables_fit(spots):
    assert check(spots, 0, 0, 0) == 0


@pytest.mark.parametrize("spots", [1, 4, 7, 10])
def test_a_word_that_leaves_its_table_is_refused(spots):
    rng = np.random.default_rng(spots)
    items = 1
    while check(spots, 0, items, 0) == 0:
        items += 1
    children = 1
    while check(spots, 1, children, 0) == 0:
        children += 1
    for at in sorted({0, items - 1, *rng.integers(0, items, 8).tolist()}):
        for delta in (1, 1 << 12, 1024 << 21):      # another item's entry or none, a subset of side 1 that is none
            assert check(spots, 0, at, delta) == PG_ERR_BOUNDS, (at, delta)
    assert check(spots, 0, 0, 255 << 13) == PG_ERR_BOUNDS   # (the first item's subset of side 0 is the first)
    for at in sorted({0, children - 1, *rng.integers(0, children, 8).tolist()}):
        assert check(spots, 1, at, 5000) == PG_ERR_BOUNDS
    assert check(spots, 2, 0, 11 << 10) == PG_ERR_BOUNDS
    for at in range(spots + 1):
        assert check(spots, 3, at, 9000) == PG_ERR_BOUNDS
        assert check(spots, 3, at, -9000) == PG_ERR_BOUNDS
