"""Short top-k lists of many rows take a form of their own: the tokens it draws are those that the same rows draw one by one (which
take the other form), at the edges of its range and for rows that its quick way must leave: ties, bans, constants, numbers that are none."""

import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab", [(18, 8000), (37, 8003), (38, 50257), (64, 151936), (70, 30011)])
@pytest.mark.parametrize("top_k,top_p,min_p", [(1, 1.0, 0.0), (2, 0.5, 0.0), (50, 0.9, 0.0), (50, 1.0, 0.05), (49, 0.8, 0.0)])
def test_rows_draw_what_they_draw_alone(rows, vocab, top_k, top_p, min_p):
    lean = kernel_ops.lib().dll.slb_sample_lean
    assert lean(rows, vocab, top_k) and not lean(1, vocab, top_k) and not lean(rows, vocab, 51) and not lean(rows, 7999, top_k) and not lean(17, vocab, top_k)
    g = torch.Generator().manual_seed(rows + top_k)
    logits = torch.randn(rows, vocab, generator=g) * 2.5
    logits[1] = 0.25                                             # all tie
    logits[2, 1000:] = float("-inf")                             # few are allowed
    logits[3, 500:7000] = -3.4028234663852886e38                 # banned
    logits[4, 77] = float("nan")
    logits[5, ::997] = 9.0                                       # ties at the top, more than the list asks for
    logits[6, 12] = float("inf")
    logits[7] = torch.arange(vocab).float().flip(0) / vocab      # the largest side by side
    logits[8, 1:] = float("-inf")
    logits[9] = torch.round(logits[9])
    logits[10, :1500] += 8.0                                     # the candidates side by side, in one block's part
    logits[11] = logits[11].sort(descending=True)[0]
    logits[12] *= 0.1
    logits[12, 4321] = 30.0                                      # one far above the others: wide steps
    logits[13] = float("-inf")
    logits[13, 5:5 + 4 * 150:4] = torch.randn(150, generator=g)  # fewer allowed than the longest lists
    logits[14] = -3.4028234663852886e38
    logits[14, 100:103] = torch.tensor([1.0, 0.5, 0.25])
    logits[15, :] = torch.linspace(1e4, 1e4 + 1.0, vocab)        # steps near the last place
    logits[16, ::2] = float("-inf")
    logits, uniform = logits.to(DEV), torch.rand(rows, generator=g).to(DEV)
    out, alone = torch.full((rows,), -1, dtype=torch.int32, device=DEV), torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    ops().sample(logits, vocab, 0.8, top_k, top_p, min_p, uniform, out)
    for r in range(rows):
        ops().sample(logits[r:r + 1], vocab, 0.8, top_k, top_p, min_p, uniform[r:r + 1], alone[r:r + 1])
    assert torch.equal(out, alone)
