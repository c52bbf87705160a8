"""The training gradient when parameters or logits are not finite: what the
oracle's gradient in double precision has as NaN or an infinity is that here
too, and a component that it has as a finite number stays one (a sample adds
to the rows of its own features only, one that does not count adds nothing).

Tolerance of the finite components: as in the gradient's other tests, 1e-4 of
the largest (fp32 sums of a few hundred terms)."""
import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu

INF, NAN = np.inf, np.nan
STONE = 18 * 2 + 2 * 4    # a black stone on the middle of quadrant 2: some nodes have it
# (parameter block, index in it, value): one each, and two together
ODD = [[("B3", 1, INF)], [("B3", 0, -INF)], [("B3", 2, NAN)], [("W3", 7, INF)], [("W3", 100, -INF)], [("W3", 100, NAN)],
       [("B2", 5, INF)], [("B2", 5, -INF)], [("B1", 9, INF)], [("B1", 9, NAN)], [("W1", STONE * 64 + 3, INF)],
       [("W1", STONE * 64 + 3, -INF)], [("W1", STONE * 64 + 3, NAN)], [("W1", STONE * 64 + 3, INF), ("B3", 1, INF)]]


@pytest.mark.parametrize("odd", ODD, ids=lambda o: " ".join(f"{b}[{i}]={v}" for b, i, v in o))
@pytest.mark.parametrize("k", [3, 700])
def test_gradient_of_parameters_that_are_not_finite(cuda, O, odd, k):
    import torch
    from pentago_b200 import capi, learned
    from pentago_b200.end import section_sig
    rng = np.random.default_rng(k)
    section, block, nodes = section_sig([[4, 4], [4, 5], [4, 3], [3, 3]]), (3, 1, 7, 9), 4096
    refs = (capi.pg_block_ref_t * 1)()
    refs[0].section = section
    for q in range(4):
        refs[0].block[q] = block[q]
    value = rng.integers(0, 3, (nodes, 1))
    sym = np.where(rng.random((nodes, 256)) < 0.3, rng.integers(0, 3, (nodes, 256)), value).astype(np.uint8).reshape(-1)
    params = (rng.standard_normal(learned.N_PARAMS) * 0.2).astype(np.float32)
    for name, i, v in odd:
        params[getattr(learned, "P_" + name) + i] = v
    samples = rng.integers(0, nodes, k).astype(np.int64) << 8 | rng.integers(0, 256, k)
    mixed = np.concatenate([samples, [1 << 24, nodes << 8 | 5, -1]])[rng.permutation(k + 3)]   # three that do not count
    tr = learned.Trainer(refs, torch.from_numpy(sym).cuda(), torch.tensor([0, 256 * nodes]).cuda(), np.array([nodes]),
                         params=torch.from_numpy(params).cuda())
    got, loss = tr.grad_of(torch.from_numpy(mixed).cuda())
    got, loss = got.cpu().numpy().astype(np.float64), float(loss.item())
    want, blk = np.zeros(learned.N_PARAMS), np.array(block, np.int32)
    wl = O.lm_grad(P(params), section, P(blk), P(sym), P(samples), k, P(want))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    fin = np.isfinite(want)
    assert np.isfinite(got[fin]).all()
    assert np.abs(got[fin] - want[fin]).max() <= 1e-4 * max(np.abs(want[fin]).max(), 1e-30)
    if np.isfinite(wl):
        assert abs(loss - wl) <= 1e-4 * abs(wl)
    else:
        assert (np.isnan(loss), loss) == (np.isnan(wl), wl) or np.isnan(loss) and np.isnan(wl)
