"""Parents are written two at a time: lines with an odd number of parents to a
CTA's microlines and with a single one, on each axis, fresh and accumulating,
with outputs at an address that allows 256-bit accesses and at one that does
not, against the oracle."""
import ctypes

import numpy as np
import pytest

from tests.oracle import P

pytestmark = pytest.mark.gpu

# sections whose four axes have 1, 3, 9, 10, 18, ... quadrants
SECTIONS = [[[9, 0], [0, 9], [5, 4], [4, 4]], [[1, 0], [0, 9], [9, 0], [4, 4]], [[0, 0], [1, 0], [0, 1], [1, 1]],
            [[4, 4], [4, 4], [5, 4], [4, 4]]]


@pytest.mark.parametrize("counts", SECTIONS)
@pytest.mark.parametrize("dim", range(4))
def test_lines_of_odd_sizes_match_oracle(cuda, O, counts, dim):
    import torch
    from pentago_b200 import end
    from pentago_b200.synthetic import random_nodes
    sig = end.section_sig(counts)
    try:
        line = end.Line(sig, dim, (0, 0, 0))
        info = end.line_info(line)
    except Exception:
        pytest.skip("no line along this axis")
    inp = random_nodes(7 * dim + 1, max(info.input_nodes, 1))
    line.input = torch.from_numpy(inp.view(np.int64)).cuda()
    want = np.zeros((info.output_nodes, 8), np.uint64)
    O.compute_line(sig, dim, line.length, (ctypes.c_uint8 * 3)(0, 0, 0), P(inp), P(want), 8)
    prior = random_nodes(99, info.output_nodes)
    for flags in (0, 1):
        for shift in (0, 2):   # 16-byte words: 32-byte aligned or not
            buf = torch.full((8 * info.output_nodes + 16,), 3, dtype=torch.int64, device="cuda")
            out = buf[shift:shift + 8 * info.output_nodes].view(-1, 8)
            out.copy_(torch.from_numpy(prior.view(np.int64)))
            line.flags, line.output = flags, out
            end.compute_lines([line])
            end.check_errors()
            got = out.cpu().numpy().view(np.uint64)
            assert np.array_equal(got, want | prior if flags else want)
            rest = torch.cat([buf[:shift], buf[shift + 8 * info.output_nodes:]])
            assert (rest == 3).all()
