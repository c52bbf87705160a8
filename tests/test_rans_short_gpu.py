"""Format-2 coding of batches of many streams, and of streams around the
lengths where the encoder's and decoder's forms change: the encoder stages
1,024 symbols at a time and leaves the counting and packing of streams above
2,048 symbols (16,384 in batches of more than 1,024 streams) to kernels of
their own; the decoder works in blocks of 1,024, and streams of up to 12,288
symbols in batches of more than 4,736 have a kernel of their own.  Streams equal the oracle's
bytes, decode to the symbols, and write nothing beside their room."""
import numpy as np
import pytest

from tests.oracle import P
from tests.test_rans_chunks_gpu import decode_bytewise, draw, oracle_encode

pytestmark = pytest.mark.gpu

EDGES = (0, 1, 8, 9, 255, 256, 511, 512, 513, 767, 768, 769, 1015, 1016, 1023, 1024, 1025, 2046, 2047, 2048, 2049, 2050, 4096,
         6143, 6145)
FAR = (8192, 12287, 12288, 12289, 16383, 16384, 16385, 20000)


def roundtrip(O, syms, align, gap, check):
    import torch
    from pentago_b200 import capi, rans
    L, k = capi.lib(), len(syms)
    n = np.array([len(s) for s in syms], np.int64)
    offsets = align + np.concatenate([[0], np.cumsum(n)])
    flat = np.concatenate([np.zeros(align, np.uint8)] + syms)
    caps = np.array([rans.bound(int(x)) for x in n], np.int64)
    at = align + np.concatenate([[0], np.cumsum(caps + gap)])
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out = torch.full((int(at[-1]) + 16,), 0xAB, dtype=torch.uint8, device="cuda")
    sizes = torch.full((k,), 777, dtype=torch.int64, device="cuda")
    d_sym, d_off, d_at, d_n = d(flat), d(offsets), d(at[:-1]), d(n)
    capi.check(L.pg_rans_encode_batch(d_sym.data_ptr(), d_off.data_ptr(), k, out.data_ptr(), d_at.data_ptr(),
                                      sizes.data_ptr(), None))
    host, sz = out.cpu().numpy(), sizes.cpu().numpy()
    for i in check:
        assert host[at[i]:at[i] + sz[i]].tobytes() == oracle_encode(O, syms[i]), (i, n[i])
    if gap:
        room = np.zeros(len(host), bool)
        for a, c in zip(at, caps):
            room[a:a + c] = True
        assert (host[~room] == 0xAB).all()
    back = torch.full((len(flat) + 16,), 0xCD, dtype=torch.uint8, device="cuda")
    status = torch.full((k,), 777, dtype=torch.int64, device="cuda")
    capi.check(L.pg_rans_decode_batch(out.data_ptr(), d_at.data_ptr(), sizes.data_ptr(), k, back.data_ptr(),
                                      d_off.data_ptr(), d_n.data_ptr(), status.data_ptr(), None))
    got = back.cpu().numpy()
    assert np.array_equal(status.cpu().numpy(), n)
    assert np.array_equal(got[align:len(flat)], flat[align:])
    assert (got[:align] == 0xCD).all() and (got[len(flat):] == 0xCD).all()


@pytest.mark.parametrize("kind", ["rare", "uniform", "skewed"])
@pytest.mark.parametrize("align", [0, 3])
def test_streams_at_the_edges_of_the_forms(cuda, O, kind, align):
    rng = np.random.default_rng(align)
    syms = [draw(rng, n, kind) for n in EDGES + FAR]
    roundtrip(O, syms, align, 3, range(len(syms)))


@pytest.mark.parametrize("kind", ["rare", "uniform"])
@pytest.mark.parametrize("count", [1024, 1025, 4736, 4737, 9000])
def test_batches_of_many_streams(cuda, O, kind, count):
    """Mostly one-node streams, with others of any length among them."""
    rng = np.random.default_rng(count)
    lengths = np.full(count, 256)
    odd = rng.permutation(count)[:200]
    lengths[odd] = rng.choice(EDGES + FAR, 200)
    syms = [draw(rng, int(n), kind) for n in lengths]
    roundtrip(O, syms, 5, 0, np.concatenate([odd, rng.integers(0, count, 20)]))


@pytest.mark.parametrize("count", [3, 1500])
def test_streams_that_cannot_be_coded(cuda, O, count):
    """A symbol above 2 anywhere refuses its stream, whoever counts it, and no other."""
    import torch
    from pentago_b200 import capi, rans
    rng = np.random.default_rng(count)
    lengths = rng.choice((0, 9, 256, 2048, 2049, 17000), count)
    lengths[:3] = (9, 2049, 17000)
    syms = [draw(rng, int(n), "uniform") for n in lengths]
    wrong = [i for i in range(count) if lengths[i] and (i < 3 or rng.random() < 0.2)]
    for i in wrong:
        syms[i][rng.choice((0, lengths[i] - 1, lengths[i] // 2))] = rng.choice((3, 4, 128, 255))
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    caps = np.array([rans.bound(int(x)) for x in lengths], np.int64)
    at = np.concatenate([[0], np.cumsum(caps)]).astype(np.int64)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out, sizes = torch.zeros(int(at[-1]), dtype=torch.uint8, device="cuda"), torch.zeros(count, dtype=torch.int64, device="cuda")
    d_sym, d_off, d_at = d(np.concatenate(syms)), d(offsets), d(at[:-1])
    capi.check(capi.lib().pg_rans_encode_batch(d_sym.data_ptr(), d_off.data_ptr(), count, out.data_ptr(), d_at.data_ptr(),
                                               sizes.data_ptr(), None))
    sz, host = sizes.cpu().numpy(), out.cpu().numpy()
    assert (sz[wrong] == -1).all()
    good = np.setdiff1d(np.arange(count), wrong)
    assert (sz[good] > 0).all()
    for i in good[:40]:
        assert host[at[i]:at[i] + sz[i]].tobytes() == oracle_encode(O, syms[i])


@pytest.mark.parametrize("kind", ["rare", "uniform"])
@pytest.mark.parametrize("damage", ["bytes", "states", "lengths"])
@pytest.mark.parametrize("others", [0, 4800])
def test_damaged_streams_in_both_forms(cuda, O, kind, damage, others):
    """Damage in streams whose symbols need one byte at most and in such that need two, in a few streams and among
    many: decoded symbol by symbol as the byte-wise rule has it, the streams beside them as they are."""
    from pentago_b200 import rans
    rng = np.random.default_rng(len(damage) + others)
    whole = [draw(rng, 256, kind) for _ in range(40)]
    good = [oracle_encode(O, s) for s in whole]
    blobs = [good[i % 40] for i in range(others)]
    for n in (300, 1500, 6007, 9000, 13000):
        blob = bytearray(oracle_encode(O, draw(rng, n, kind)))
        lens = np.frombuffer(bytes(blob[28:60]), "<u4").astype(np.int64)
        if damage == "bytes":
            for k in rng.integers(60, len(blob), 20):
                blob[k] ^= int(rng.integers(1, 256))
        elif damage == "states":
            starts = 60 + np.concatenate([[0], np.cumsum(lens)[:-1]])
            for k, v in zip(starts, (bytes(4), b"\0\0\0\1", b"\0\x7f\xff\xff", b"\xff" * 4, b"\x80\0\0\0")):
                blob[int(k):int(k) + 4] = v
        else:
            lens[0] -= 1
            lens[1] += 1
            lens[7] += lens[6] - 2
            lens[6] = 2
            blob[28:60] = lens.astype("<u4").tobytes()
        at = int(rng.integers(0, len(blobs) + 1))
        blobs.insert(at, bytes(blob))
    for k, (blob, got) in enumerate(zip(blobs, rans.decode(blobs))):
        want = [whole[i] for i in range(40) if good[i] is blob] or [decode_bytewise(blob)]
        assert np.array_equal(got, want[0]), k
