"""Blocks that the store coder keeps raw, in streams at every alignment: the
nodes lie where the stream starts, which need not be an 8-byte boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = np.array([1, 2, 31, 33, 65, 300], np.int32)


@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4, 6, 8])
@pytest.mark.parametrize("turn", [0, 1])
def test_raw_blocks_at_any_alignment(cuda, turn, shift):
    import torch
    from pentago_b200 import capi
    from pentago_b200.slice_store import store_bound
    L, n, k = capi.lib(), int(COUNTS.sum()), len(COUNTS)
    rng = np.random.default_rng(10 * shift + turn)
    win = rng.integers(0, 1 << 64, (n, 4), dtype=np.uint64)
    nodes = np.concatenate([win, win | rng.integers(0, 1 << 64, (n, 4), dtype=np.uint64)], 1)
    # a table that expects symbol 0 everywhere: two symbols in three cost 14 bits
    table = torch.tensor([16382, 1, 1] * 1024, dtype=torch.int16, device="cuda")
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    first, count = np.concatenate([[0], np.cumsum(COUNTS)[:-1]]).astype(np.int64), COUNTS
    caps = (store_bound(COUNTS) + 15) // 16 * 16
    off = np.concatenate([[0], np.cumsum(caps)])[:-1].astype(np.int64) + shift
    out = torch.full((int(caps.sum()) + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(k, dtype=torch.int64, device="cuda")
    d_nodes, d_first, d_count, d_off = d(nodes.view(np.int64)), d(first), d(count), d(off)
    capi.check(L.pg_store_encode(d_nodes.data_ptr(), d_first.data_ptr(), d_count.data_ptr(), k, turn, table.data_ptr(),
                                 out.data_ptr(), d_off.data_ptr(), sizes.data_ptr(), None))
    host = out.cpu().numpy()
    assert sizes.cpu().tolist() == (128 + 64 * COUNTS).tolist()
    for o, f, c in zip(off, first, COUNTS):
        assert host[o:o + 4].tolist() == [255] * 4 and not host[o + 4:o + 128].any()
        assert host[o + 128:o + 128 + 64 * c].tobytes() == nodes[f:f + c].tobytes()
    assert (host[:shift] == 0xAB).all() and (host[int(off[-1] + caps[-1]):] == 0xAB).all()
    back, status = torch.zeros_like(d_nodes), torch.zeros(k, dtype=torch.int64, device="cuda")
    capi.check(L.pg_store_decode(out.data_ptr(), d_off.data_ptr(), sizes.data_ptr(), d_count.data_ptr(),
                                 d_first.data_ptr(), k, turn, table.data_ptr(), back.data_ptr(), status.data_ptr(),
                                 None))
    assert status.cpu().tolist() == COUNTS.tolist()
    assert torch.equal(back, d_nodes)
