"""Midsolve of mixed batches at the edges of its row tables: every number of
stones a side may have, the first and last board that one CTA solves alone, and
boards large enough that a group's share of a level is several chunks.  The
values are whole numbers, so they are the oracle's exactly."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu


def oracle_values(O, raw):
    r, v = np.zeros(200, np.uint64), np.zeros(200, np.int32)
    n = O.midsolve(int(raw), P(r), P(v))
    return list(zip(r[:n].tolist(), v[:n].tolist()))


@pytest.mark.parametrize("stones", [(36, 35, 34, 32, 26, 25), (27, 22, 26), (21,)])
def test_mixed_batch_matches_oracle(cuda, O, stones):
    from pentago_b200 import mid
    raws = np.concatenate([mid.random_boards(300 + s, 1, s) for s in stones])
    raws = np.concatenate([raws, raws[::-1] | np.uint64(1 << 63)])
    for raw, g in zip(raws, mid.midsolve(raws)):
        assert g == oracle_values(O, raw), f"board {int(raw)}"


def test_more_small_boards_than_fit_at_once(cuda, O):
    """Every size of board that is solved over index tables, in a batch of
    more cluster pairs than the GPU holds at once."""
    from pentago_b200 import mid
    raws = np.concatenate([mid.random_boards(400 + s, 30 if s > 28 else 3, s) for s in range(26, 37)])
    raws[1::2] |= np.uint64(1 << 63)
    for raw, g in zip(raws, mid.midsolve(raws)):
        assert g == oracle_values(O, raw), f"board {int(raw)}"
