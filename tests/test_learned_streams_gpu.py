"""Learned coder streams at the edges of its kernels: one node, runs of one
node with idle lanes, exactly 32 nodes, several rounds, an odd number of
streams, symbols at an odd address, and models whose frequencies are extreme
(activations past their cut, probabilities below the smallest).  Streams are
defined bit by bit, so they equal the oracle's bytes and decode to the
symbols."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu

# section, block, nodes
BLOCKS = [([[0, 0], [0, 0], [0, 0], [0, 0]], (0, 0, 0, 0), 1), ([[0, 0], [0, 0], [1, 0], [0, 1]], (0, 0, 0, 0), 9),
          ([[0, 0], [1, 1], [1, 1], [1, 1]], (0, 0, 2, 2), 32), ([[0, 0], [1, 0], [1, 0], [0, 1]], (0, 0, 0, 0), 27),
          ([[0, 0], [0, 0], [1, 1], [1, 1]], (0, 0, 0, 0), 64), ([[1, 0], [0, 1], [1, 1], [1, 1]], (0, 0, 2, 2), 36),
          ([[1, 0], [1, 0], [0, 1], [0, 1]], (0, 0, 0, 0), 81), ([[1, 0], [1, 1], [1, 1], [1, 1]], (0, 0, 0, 2), 384),
          ([[0, 0], [0, 0], [0, 0], [1, 1]], (0, 0, 0, 0), 8)]


def predictor(scale, rng):
    """A model that expects a symbol to be its neighbours' and the previous node's."""
    from pentago_b200 import learned
    p = np.zeros(learned.N_PARAMS, np.float32)
    w1, w2 = rng.standard_normal((124, 64)) * 0.05, rng.standard_normal((64, 64)) * 0.05
    w3 = rng.standard_normal((64, 3)) * 0.05
    for v in range(3):
        w1[88 + v:120:4, v] += 0.5 * scale
        w1[120 + v, v] += 1.5 * scale
        w2[v, v] += scale
        w3[v, v] += scale
    p[learned.P_W1:learned.P_B1], p[learned.P_W2:learned.P_B2] = w1.reshape(-1), w2.reshape(-1)
    p[learned.P_W3:learned.P_B3] = w3.reshape(-1)
    p[learned.P_B3:learned.P_B3 + 3] = rng.standard_normal(3) * 0.2
    model = np.zeros(learned.model_bytes(), np.uint8)
    from pentago_b200 import capi
    capi.check(capi.lib().pg_learned_export(P(p), P(model)))
    return model.tobytes()


@pytest.mark.parametrize("scale,picks", [(1, range(9)), (4, range(9)), (12, range(9)), (1, [7]), (4, [3, 0]), (12, [0])])
def test_edge_streams_match_oracle_bytes(cuda, O, scale, picks):
    import torch
    from pentago_b200 import capi, learned
    from pentago_b200.end import section_sig
    rng = np.random.default_rng(100 * scale + len(picks))
    model = predictor(scale, rng)
    refs = (capi.pg_block_ref_t * len(picks))()
    for ref, b in zip(refs, picks):
        ref.section = section_sig(BLOCKS[b][0])
        for q in range(4):
            ref.block[q] = BLOCKS[b][1][q]
    nodes = np.array([BLOCKS[b][2] for b in picks], np.int64)
    offsets = np.concatenate([[0], np.cumsum(256 * nodes)])
    # a value per node: what the model predicts and the format-2 coder cannot
    sym = np.repeat(rng.integers(0, 3, int(nodes.sum())), 256).astype(np.uint8)
    noise = rng.random(len(sym)) < 0.02
    sym[noise] = rng.integers(0, 3, int(noise.sum()))
    odd = torch.from_numpy(np.concatenate([[9], sym]).astype(np.uint8)).cuda()[1:]
    data, doff, dsz = learned.encode(model, refs, odd, torch.from_numpy(offsets).cuda(), nodes)
    host, hoff, hsz = data.cpu().numpy(), doff.cpu().numpy(), dsz.cpu().numpy()
    mbytes = np.frombuffer(model, np.uint8)
    learned_streams = 0
    for s in range(len(picks)):
        mine, blk = np.ascontiguousarray(sym[offsets[s]:offsets[s + 1]]), np.array(list(refs[s].block), np.int32)
        lm, st = np.zeros(200 + 2 * mine.size, np.uint8), np.zeros(mine.size // 4 + 1000, np.uint8)
        n = O.lm_encode(P(mbytes), refs[s].section, P(blk), P(mine), P(lm), lm.size)
        m = O.rans_encode(P(mine), mine.size, P(st), st.size)
        assert n > 0 and m > 0
        learned_streams += n <= m
        assert host[hoff[s]:hoff[s] + hsz[s]].tobytes() == (lm[:n] if n <= m else st[:m]).tobytes()
    assert learned_streams or len(picks) < 3
    got, _, status = learned.decode(model, refs, data, doff, dsz, nodes)
    assert status.cpu().tolist() == (256 * nodes).tolist()
    assert np.array_equal(got.cpu().numpy(), sym)
