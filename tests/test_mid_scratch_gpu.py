"""Midsolve batches in exactly the scratch that they ask for: the results of the
allocating call, and nothing written past the buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stones", [(36,), (26,) * 9, (30, 25, 26), (24, 27, 22, 33)])
def test_batches_in_the_scratch_they_ask_for(cuda, stones):
    import torch
    from pentago_b200 import capi, mid
    raws = np.concatenate([mid.random_boards(7 + k, 1, s) for k, s in enumerate(stones)])
    need = mid.scratch_bytes(raws)
    scratch = torch.full((need + 4096,), 0xAB, dtype=torch.uint8, device="cuda")
    out = torch.zeros((len(raws), mid.RECORD_BYTES), dtype=torch.uint8, device="cuda")
    capi.check(capi.lib().pg_midsolve_batch(capi.ptr(raws), len(raws), out.data_ptr(), scratch.data_ptr(), need, None))
    assert mid.decode(out.cpu().numpy()) == mid.midsolve(raws)
    assert (scratch[need:] == 0xAB).all()
    assert capi.lib().pg_midsolve_batch(capi.ptr(raws), len(raws), out.data_ptr(), scratch.data_ptr(), need - 1, None) < 0
