"""The sampler's quick path (one read of the row, one histogram of values; csrc/sampling.cu) against its general path, which takes
any row: the same logits with finite, hopeless tokens behind them, so many that the blocks cannot hold the row."""

import numpy as np
import pytest
import torch

from sleuth_b200.sampling.config import SamplingConfig
from sleuth_b200.sampling.sampler import Sampler

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HELD = 8 * 20480        # tokens of a row that a team of eight blocks holds


def rows_of(kind, vocab, gen):
    x = torch.randn((6, vocab), generator=gen) * 2.5
    if kind == "ties":                                    # many equal values, also at every threshold
        x = (x * 2).round() / 2
    elif kind == "banned":
        x[:, ::3] = -3.4028234663852886e38
    elif kind == "flat":
        x[:3] = 1.25
    elif kind == "shifted":
        x += 40.0
    elif kind == "masked":                                # whole stretches are -inf: the quick path must decline
        x[:, vocab // 4: vocab - vocab // 4] = float("-inf")
    elif kind == "peak":
        x[torch.arange(6), torch.randint(0, vocab, (6,), generator=gen)] = 60.0
    return x


# 503: one warp of some blocks holds anything; 50,257: rows that start off a 16-byte boundary; the largest row that is held.
@pytest.mark.parametrize("vocab", [503, 4096, 50257, 151936, HELD])
@pytest.mark.parametrize("kind", ["normal", "ties", "banned", "flat", "shifted", "masked", "peak"])
def test_quick_and_general_path_choose_the_same_tokens(vocab, kind):
    gen = torch.Generator().manual_seed(vocab + len(kind))
    x = rows_of(kind, vocab, gen)
    quick = x.to(DEV)
    general = torch.full((6, HELD + 8), -1e30)
    general[:, :vocab] = x
    general = general.to(DEV)
    u = np.random.default_rng(vocab).random((4, 6), dtype=np.float32)
    u[0, 0], u[0, 1] = 0.0, np.nextafter(np.float32(1), np.float32(0))
    for k, p, m in [(1, 1.0, 0.0), (5, 1.0, 0.05), (50, 0.9, 0.0), (50, 0.3, 0.0), (400, 1.0, 0.0), (400, 0.98, 0.05), (1500, 0.9, 0.0),
                    (0, 0.7, 0.0), (0, 0.98, 0.0), (0, 1e-6, 0.0), (0, 0.9, 0.1), (vocab - 1, 0.9, 0.0)]:
        for t in (0.5, 0.8, 1.2, 40.0):
            cfg = SamplingConfig(temperature=t, top_k=k, top_p=p, min_p=m)
            for uu in u[:2 if t != 0.8 else 4]:
                a = Sampler(DEV, vocab).choose(quick, cfg, uu).clone()
                b = Sampler(DEV, HELD + 8).choose(general, cfg, uu)
                assert torch.equal(a, b), (k, p, m, t, a.tolist(), b.tolist())
