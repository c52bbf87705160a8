"""Learned coder: a tensor-core product whose wait runs out is reported for
every stream that it concerns, also when it is a stream's last one, and for the
streams that no CTA came to (their sizes and statuses are not what the arrays
held before).  The wait is taken to have run out; nothing is left in flight."""
import numpy as np
import pytest

from tests.test_learned_streams_gpu import BLOCKS, predictor

pytestmark = pytest.mark.gpu

PG_ERR_CUDA = -2


@pytest.mark.parametrize("picks", [[1], list(range(9)), [1] * 2000])
def test_unfinished_products_are_reported(cuda, picks):
    import torch
    from pentago_b200 import capi, learned
    from pentago_b200.end import section_sig
    rng, L = np.random.default_rng(len(picks)), capi.lib()
    model = predictor(1, rng)
    refs = (capi.pg_block_ref_t * len(picks))()
    for ref, b in zip(refs, picks):
        ref.section = section_sig(BLOCKS[b][0])
        for q in range(4):
            ref.block[q] = BLOCKS[b][1][q]
    nodes = np.array([BLOCKS[b][2] for b in picks], np.int64)
    offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(256 * nodes)])).cuda()
    sym = torch.from_numpy(np.repeat(rng.integers(0, 3, int(nodes.sum())), 256).astype(np.uint8)).cuda()
    data, doff, dsz = learned.encode(model, refs, sym, offsets, nodes)
    out, sizes = torch.zeros_like(data), torch.full_like(dsz, 777)
    capi.check(L.pg_debug_learned_encode(learned._model_ptr(model), refs, len(refs), sym.data_ptr(), offsets.data_ptr(),
                                         out.data_ptr(), doff.data_ptr(), sizes.data_ptr(), None))
    assert (sizes == PG_ERR_CUDA).all()
    version = data[doff[:-1]]          # the streams' first bytes
    assert (version == 3).any()
    back, status = torch.zeros_like(sym), torch.full_like(dsz, 777)
    caps = torch.from_numpy(256 * nodes).cuda()
    capi.check(L.pg_debug_learned_decode(learned._model_ptr(model), refs, len(refs), data.data_ptr(), doff.data_ptr(),
                                         dsz.data_ptr(), back.data_ptr(), offsets.data_ptr(), caps.data_ptr(),
                                         status.data_ptr(), None))
    assert torch.equal(status, torch.where(version == 3, torch.full_like(caps, PG_ERR_CUDA), caps))
    # and the next calls are as they were
    again, _, asz = learned.encode(model, refs, sym, offsets, nodes)
    assert torch.equal(asz, dsz)
    back, _, status = learned.decode(model, refs, again, doff, asz, nodes)
    assert torch.equal(back, sym) and torch.equal(status, caps)
