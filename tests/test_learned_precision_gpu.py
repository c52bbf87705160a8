"""The training gradient's precision: its error against the oracle's gradient in
double precision, as a part of the gradient's norm.

Tolerance 3e-7.  The kernel's products are exact and its sums are of fp32 values,
each addition rounded to 2^-24: with loops over the samples in fp32 the error
is 1.0e-7 to 2.1e-7 of the norm at such batches.  Sums that the tensor cores
join themselves drop bits and come to 3.9e-7, gradients without the third of
their bf16 terms to 2^-17, about 8e-6; either is refused here."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [3000, 40000])
def test_gradient_error_as_a_part_of_its_norm(cuda, O, k):
    import torch
    from pentago_b200 import capi, learned
    from pentago_b200.end import section_sig
    rng = np.random.default_rng(k + 1)
    section, block, nodes = section_sig([[4, 4], [4, 5], [4, 3], [3, 3]]), (3, 1, 7, 9), 4096
    refs = (capi.pg_block_ref_t * 1)()
    refs[0].section = section
    for q in range(4):
        refs[0].block[q] = block[q]
    value = rng.integers(0, 3, (nodes, 1))
    sym = np.where(rng.random((nodes, 256)) < 0.3, rng.integers(0, 3, (nodes, 256)), value).astype(np.uint8).reshape(-1)
    params = (rng.standard_normal(learned.N_PARAMS) * 0.15).astype(np.float32)
    samples = rng.integers(0, nodes, k).astype(np.int64) << 8 | rng.integers(0, 256, k)
    tr = learned.Trainer(refs, torch.from_numpy(sym).cuda(), torch.tensor([0, 256 * nodes]).cuda(), np.array([nodes]),
                         params=torch.from_numpy(params).cuda())
    got, loss = tr.grad_of(torch.from_numpy(samples).cuda())
    got = got.cpu().numpy().astype(np.float64)
    want, blk = np.zeros(learned.N_PARAMS), np.array(block, np.int32)
    wl = O.lm_grad(P(params), section, P(blk), P(sym), P(samples), k, P(want))
    error = np.linalg.norm(got - want) / np.linalg.norm(want)
    print(f"error {error:.2e} of the norm")
    assert error <= 3e-7
    assert abs(float(loss.item()) - wl) <= 1e-6 * abs(wl)
