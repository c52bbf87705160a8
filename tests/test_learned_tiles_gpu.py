"""The training gradient at the edges of its kernel's tiles (16 samples to a
warp, 224 to a CTA, more tiles than CTAs), with samples that do not count
among them, against the oracle's gradient in double precision.

Tolerance: a component is a sum over samples in fp32, at most 42 tensor-core
steps and a few hundred additions deep, each off by at most 2^-22 of the
partial sum: 1e-4 of the largest component leaves room for cancellation."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 15, 16, 17, 223, 224, 225, 3000, 40000])
def test_gradient_at_tile_edges(cuda, O, k):
    import torch
    from pentago_b200 import capi, learned
    from pentago_b200.end import section_sig
    rng = np.random.default_rng(k)
    section = section_sig([[4, 4], [4, 5], [4, 3], [3, 3]])
    refs = (capi.pg_block_ref_t * 2)()
    for b, block in enumerate(((3, 1, 7, 9), (19, 4, 39, 52))):     # a full block, a ragged one (8 x 2 x 6 x 4)
        refs[b].section = section
        for q in range(4):
            refs[b].block[q] = block[q]
    nodes = np.array([4096, 8 * 2 * 6 * 4])
    value = rng.integers(0, 3, (int(nodes.sum()), 1))
    sym = np.where(rng.random((int(nodes.sum()), 256)) < 0.3, rng.integers(0, 3, (int(nodes.sum()), 256)), value)
    sym = sym.astype(np.uint8).reshape(-1)
    offsets = np.concatenate([[0], np.cumsum(256 * nodes)])
    params = (rng.standard_normal(learned.N_PARAMS) * 0.2).astype(np.float32)
    s = rng.integers(0, 2, k)
    local = rng.integers(0, nodes[s]) << 8 | rng.integers(0, 256, k)
    samples = s.astype(np.int64) << 24 | local
    mixed = np.concatenate([samples, [2 << 24, 1 << 24 | int(nodes[1]) << 8 | 5, -1]])   # three that do not count
    mixed = mixed[rng.permutation(len(mixed))]
    tr = learned.Trainer(refs, torch.from_numpy(sym).cuda(), torch.from_numpy(offsets).cuda(), nodes,
                         params=torch.from_numpy(params).cuda())
    got, loss = tr.grad_of(torch.from_numpy(mixed).cuda())
    got = got.cpu().numpy().astype(np.float64)
    want, wl = np.zeros(learned.N_PARAMS), 0.0
    for b in range(2):
        mine = np.ascontiguousarray(local[s == b])
        if len(mine):
            part, blk = np.zeros(learned.N_PARAMS), np.array(list(refs[b].block), np.int32)
            host = np.ascontiguousarray(sym[offsets[b]:offsets[b + 1]])
            wl += O.lm_grad(P(params), section, P(blk), P(host), P(mine), len(mine), P(part))
            want += part
    assert abs(float(loss.item()) - wl) <= 1e-4 * abs(wl)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    again, _ = tr.grad_of(torch.from_numpy(mixed).cuda())
    assert np.array_equal(again.cpu().numpy().astype(np.float64), got)     # fixed order
