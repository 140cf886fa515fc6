"""The general attention kernel (csrc/attention_generic.cu) at the edges of its channels a lane and of the batches in which it asks
for value rows, and that no width pays for its batches with the blocks that fit an SM."""

import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, make_cache, ops, tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,number", [(torch.float32, 0), (torch.bfloat16, 1)])
def test_blocks_an_sm(dtype, number):
    """With registers for one value row at a time 3 blocks (float32, 256 channels) to 5 fit."""
    blocks = ops().lib().dll.slb_attention_generic_blocks_per_sm
    assert all(blocks(width, number) >= 4 for width in (24, 64, 80, 96, 128))
    assert blocks(128, 1) >= 5 and blocks(256, number) >= (3 if number == 0 else 4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 200, 256])
def test_value_widths(dtype, width):
    heads, kv_heads, hd = 4, 2, 48
    pasts, counts = [0, 6, 70, 255], [9, 1, 34, 2]
    gen = torch.Generator().manual_seed(width)
    lens = [p + c for p, c in zip(pasts, counts)]
    k_pool, _, table, ks, _ = make_cache(lens, kv_heads, hd, dtype, gen)
    gen.manual_seed(width)
    _, v_pool, again, _, vs = make_cache(lens, kv_heads, width, dtype, gen)
    assert torch.equal(table, again)
    q = torch.randn(sum(counts), heads, hd, generator=gen).to(dtype)
    seq, pos = np.repeat(np.arange(4), counts), np.concatenate([np.arange(p, p + c) for p, c in zip(pasts, counts)])
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32)).to(DEV)
    for window in (0, 20):
        out = torch.full((len(seq), heads * width), float("nan"), dtype=dtype, device=DEV)
        ops().attention(q.to(DEV), k_pool.to(DEV), v_pool.to(DEV), out, d(seq), d(pos), table.to(DEV), heads, kv_heads, hd, window, hd ** -0.5, value_dim=width)
        for t in range(len(seq)):
            lo = max(0, pos[t] - window + 1) if window else 0
            k, v = (a[seq[t]][lo:pos[t] + 1].double().repeat_interleave(2, 1) for a in (ks, vs))
            p = torch.softmax(torch.einsum("hd,jhd->hj", q[t].double(), k) / math.sqrt(hd), 1)
            torch.testing.assert_close(out[t].cpu().double().view(heads, width), torch.einsum("hj,jhd->hd", p, v), **tol(dtype))
