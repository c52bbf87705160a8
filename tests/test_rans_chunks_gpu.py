"""The format-2 coder kernels at the edges of their staging: streams around the
encoder's 512-symbol chunks and the decoder's 256-symbol blocks, at every
16-byte alignment of symbols and streams, in batches of unequal lengths, and
decoding of damaged streams symbol by symbol as the byte-wise rule has it."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 7, 8, 9, 255, 256, 257, 503, 511, 512, 513, 520, 1023, 1025, 2048, 4095, 6007, 20000)


def oracle_encode(O, sym):
    cap = 2 * len(sym) + 1000
    out = np.zeros(cap, np.uint8)
    n = O.rans_encode(P(sym), len(sym), P(out), cap)
    assert n > 0
    return out[:n].tobytes()


def draw(rng, n, kind):
    if kind == "rare":      # frequencies near 1: two-byte renormalizations
        return np.where(rng.random(n) < 0.999, 2, rng.integers(0, 3, n)).astype(np.uint8)
    if kind == "uniform":
        return rng.integers(0, 3, n).astype(np.uint8)
    return np.where(rng.random(n) < 0.9, 1, rng.integers(0, 3, n)).astype(np.uint8)


@pytest.mark.parametrize("kind", ["rare", "uniform", "skewed"])
@pytest.mark.parametrize("align", [0, 1, 5, 15])
def test_batches_of_unequal_streams(cuda, O, kind, align):
    import torch
    from pentago_b200 import capi, rans
    rng = np.random.default_rng(align)
    syms = [draw(rng, n, kind) for n in LENGTHS]
    blobs = [oracle_encode(O, s) for s in syms]
    offsets = np.cumsum([align] + [len(s) for s in syms]).astype(np.int64)
    flat = np.concatenate([np.zeros(align, np.uint8)] + syms)
    # encode with streams placed at odd offsets of the output
    caps = np.array([rans.bound(len(s)) for s in syms], np.int64)
    at = np.concatenate([[align], align + np.cumsum(caps + 3)])
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out = torch.full((int(at[-1]) + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    sizes = torch.zeros(len(syms), dtype=torch.int64, device="cuda")
    sym_d, off_d, at_d = d(flat), d(offsets), d(at[:-1].astype(np.int64))
    capi.check(capi.lib().pg_rans_encode_batch(sym_d.data_ptr(), off_d.data_ptr(), len(syms), out.data_ptr(),
                                               at_d.data_ptr(), sizes.data_ptr(), None))
    host, sz = out.cpu().numpy(), sizes.cpu().numpy()
    for i, b in enumerate(blobs):
        assert host[at[i]:at[i] + sz[i]].tobytes() == b, (kind, align, LENGTHS[i])
        assert (host[at[i] + caps[i]:at[i + 1]] == 0xAB).all()      # nothing past a stream's room
    assert (host[:align] == 0xAB).all()
    # decode at the same odd offsets, into the same odd symbol offsets
    back = torch.full((len(flat) + 16,), 0xCD, dtype=torch.uint8, device="cuda")
    n_d, status = d(np.array([len(s) for s in syms], np.int64)), torch.zeros(len(syms), dtype=torch.int64, device="cuda")
    capi.check(capi.lib().pg_rans_decode_batch(out.data_ptr(), at_d.data_ptr(), sizes.data_ptr(), len(syms),
                                               back.data_ptr(), off_d.data_ptr(), n_d.data_ptr(), status.data_ptr(), None))
    got = back.cpu().numpy()
    assert np.array_equal(got[align:len(flat)], flat[align:])
    assert (got[:align] == 0xCD).all() and (got[len(flat):] == 0xCD).all()
    assert status.cpu().tolist() == [len(s) for s in syms]


def decode_bytewise(blob):
    """Format 2 by its definition: a lane takes bytes while its state is below 2^23 and it has any left."""
    counts = [int(x) for x in np.frombuffer(blob[4:28], "<u8")]
    lens = np.frombuffer(blob[28:60], "<u4").astype(int)
    n, total = sum(counts), 1 << 14
    f = [max(1, c * total // n) for c in counts]
    f[int(np.argmax(f))] += total - sum(f)
    cum = [0, f[0], f[0] + f[1]]
    out, start = np.zeros(n, np.uint8), 60
    for lane in range(8):
        data, start = blob[start:start + lens[lane]], start + lens[lane]
        x, p = int.from_bytes(data[:4], "big"), min(4, len(data))
        for i in range(lane, n, 8):
            slot = x & (total - 1)
            s = 0 if slot < cum[1] else 1 if slot < cum[2] else 2
            x = (f[s] * (x >> 14) + slot - cum[s]) & 0xFFFFFFFF
            while x < 1 << 23 and p < len(data):
                x, p = (x << 8 | data[p]) & 0xFFFFFFFF, p + 1
            out[i] = s
    return out


@pytest.mark.parametrize("damage", ["bytes", "states", "lengths"])
def test_damaged_streams_decode_as_the_rule_says(cuda, O, damage):
    from pentago_b200 import rans
    rng = np.random.default_rng(3)
    blobs = []
    for n in (300, 6007, 9000):
        blob = bytearray(oracle_encode(O, draw(rng, n, "uniform")))
        lens = np.frombuffer(bytes(blob[28:60]), "<u4").astype(np.int64)
        if damage == "bytes":
            for k in rng.integers(60, len(blob), 40):
                blob[k] ^= int(rng.integers(1, 256))
        elif damage == "states":     # initial states below 2^23, zero, and above 2^31
            starts = 60 + np.concatenate([[0], np.cumsum(lens)[:-1]])
            for k, v in zip(starts, (bytes(4), b"\0\0\0\1", b"\0\x7f\xff\xff", b"\xff" * 4, b"\x80\0\0\0")):
                blob[int(k):int(k) + 4] = v
        else:                        # lanes of other lengths, the sum kept
            lens[0] -= 3
            lens[1] += 3
            lens[7] += lens[6] - 2
            lens[6] = 2
            blob[28:60] = lens.astype("<u4").tobytes()
        blobs.append(bytes(blob))
    for blob, got in zip(blobs, rans.decode(blobs)):
        assert np.array_equal(got, decode_bytewise(blob))


@pytest.mark.parametrize("align", [0, 1, 8])
def test_node_symbols_at_any_alignment(cuda, align):
    import torch
    from pentago_b200 import capi
    from pentago_b200.synthetic import random_nodes
    nodes = random_nodes(5, 37)
    d = torch.from_numpy(nodes.view(np.int64)).cuda()
    out = torch.full((37 * 256 + 32,), 7, dtype=torch.uint8, device="cuda")
    capi.check(capi.lib().pg_node_symbols(d.data_ptr(), 37, 1, out.data_ptr() + align, None))
    bits = lambda w: np.unpackbits(w.view(np.uint8).reshape(-1, 32), axis=1, bitorder="little")
    want = (1 - bits(nodes[:, 4:].copy()) + 2 * bits(nodes[:, :4].copy())).astype(np.uint8).reshape(-1)
    got = out.cpu().numpy()
    assert np.array_equal(got[align:align + 37 * 256], want)
    assert (got[:align] == 7).all() and (got[align + 37 * 256:] == 7).all()
