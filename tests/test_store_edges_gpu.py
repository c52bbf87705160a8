"""The store coder kernels where their forms divide: streams at offsets that
are not word aligned, nodes that are 8- but not 16-byte aligned, blocks
around the 32-lane split, and streams whose lanes a coder did not leave as
they are, which are decoded byte by byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = np.array([1, 2, 31, 32, 33, 63, 65, 255, 1024, 4096], np.int32)


def table_and_nodes(turn, seed, pad):
    """Skewed nodes starting `pad` words into their buffer, and the batch's table."""
    import torch
    from pentago_b200 import capi
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = int(COUNTS.sum())
    r = lambda: torch.randint(-2**63, 2**63 - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    x = r()
    win = x & r() & r()
    flat = torch.zeros(8 * n + 8, dtype=torch.int64, device="cuda")
    flat[pad:pad + 8 * n] = torch.cat([win, win | (x & r())], 1).reshape(-1)
    first = torch.from_numpy(np.concatenate([[0], np.cumsum(COUNTS)[:-1]]).astype(np.int64)).cuda()
    count = torch.from_numpy(COUNTS).cuda()
    table = torch.empty(3072, dtype=torch.int16, device="cuda")
    capi.check(capi.lib().pg_store_table(flat.data_ptr() + 8 * pad, first.data_ptr(), count.data_ptr(), len(COUNTS),
                                         turn, table.data_ptr(), None))
    return flat, first, count, table


def encode(flat, pad, first, count, table, turn, shift):
    import torch
    from pentago_b200 import capi
    from pentago_b200.slice_store import store_bound
    caps = (store_bound(COUNTS) + 15) // 16 * 16
    off = np.concatenate([[0], np.cumsum(caps)])[:-1] + shift
    out = torch.full((int(caps.sum()) + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(len(COUNTS), dtype=torch.int64, device="cuda")
    d_off = torch.from_numpy(off).cuda()
    capi.check(capi.lib().pg_store_encode(flat.data_ptr() + 8 * pad, first.data_ptr(), count.data_ptr(), len(COUNTS),
                                          turn, table.data_ptr(), out.data_ptr(), d_off.data_ptr(), sizes.data_ptr(),
                                          None))
    return out, off, sizes.cpu().numpy()


def decode(data, off, sizes, first, count, table, turn, pad, n):
    import torch
    from pentago_b200 import capi
    back = torch.zeros(8 * n + 8, dtype=torch.int64, device="cuda")
    status = torch.zeros(len(sizes), dtype=torch.int64, device="cuda")
    d_off, d_sz = torch.from_numpy(off).cuda(), torch.from_numpy(np.asarray(sizes, np.int64)).cuda()
    capi.check(capi.lib().pg_store_decode(data.data_ptr(), d_off.data_ptr(), d_sz.data_ptr(), count.data_ptr(),
                                          first.data_ptr(), len(sizes), turn, table.data_ptr(),
                                          back.data_ptr() + 8 * pad, status.data_ptr(), None))
    return back, status.cpu().numpy()


@pytest.mark.parametrize("turn", [0, 1])
def test_unaligned_streams_and_nodes(cuda, turn):
    import torch
    n = int(COUNTS.sum())
    flat, first, count, table = table_and_nodes(turn, 11, 0)
    out, off, sizes = encode(flat, 0, first, count, table, turn, 0)
    want = [out[o:o + s].cpu().numpy().tobytes() for o, s in zip(off, sizes)]
    flat1, _, _, table1 = table_and_nodes(turn, 11, 1)
    assert torch.equal(table, table1)
    for pad, shift in ((0, 1), (1, 0), (1, 3), (0, 2)):
        nodes = flat1 if pad else flat
        out2, off2, sizes2 = encode(nodes, pad, first, count, table, turn, shift)
        assert sizes2.tolist() == sizes.tolist()
        assert [out2[o:o + s].cpu().numpy().tobytes() for o, s in zip(off2, sizes2)] == want
        back, status = decode(out2, off2, sizes2, first, count, table, turn, pad, n)
        assert status.tolist() == COUNTS.tolist()
        assert torch.equal(back, nodes)


def test_lanes_no_coder_leaves(cuda):
    """An empty lane's final state written in three bytes decodes (its leading
    byte is zero), a lane with a state below 2^23 or with bytes missing or
    left over is refused, and the blocks beside it are not touched."""
    import torch
    turn, n = 1, int(COUNTS.sum())
    flat, first, count, table = table_and_nodes(turn, 12, 0)
    out, off, sizes = encode(flat, 0, first, count, table, turn, 0)
    host = out.cpu().numpy()
    blobs = [host[o:o + s].copy() for o, s in zip(off, sizes)]

    def run(changed):
        at = np.cumsum([0] + [(len(b) + 31) // 16 * 16 for b in changed])[:-1].astype(np.int64)
        data = np.zeros(int(at[-1]) + len(changed[-1]) + 32, np.uint8)
        for a, b in zip(at, changed):
            data[a:a + len(b)] = b
        return decode(torch.from_numpy(data).cuda(), at, [len(b) for b in changed], first, count, table, turn, 0, n)
    lens = blobs[0][:128].view("<u4")     # the one-node block: lane 0 codes it, 31 lanes are empty
    assert lens[31] == 4 and blobs[0][-4:].tolist() == [0, 0x80, 0, 0]
    short = np.concatenate([blobs[0][:-4], blobs[0][-3:]])
    short[124:128] = np.array([3], "<u4").view(np.uint8)
    back, status = run([short] + blobs[1:])
    assert status.tolist() == COUNTS.tolist() and torch.equal(back, flat)
    low = blobs[8].copy()
    low[128:132] = (0, 0, 0, 9)                     # lane 0's state
    gone = np.concatenate([blobs[9][:-1], []]).astype(np.uint8)
    gone[124:128] = (gone[124:128].view("<u4") - 1).view(np.uint8)
    more = np.concatenate([blobs[7], [0]]).astype(np.uint8)
    more[124:128] = (more[124:128].view("<u4") + 1).view(np.uint8)
    back, status = run(blobs[:7] + [more, low, gone])
    assert status.tolist()[:7] == COUNTS.tolist()[:7] and (status[7:] < 0).all()
    k = 8 * int(COUNTS[:7].sum())
    assert torch.equal(back[:k], flat[:k])
