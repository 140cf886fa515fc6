"""The sampler with few rows (blocks of 1,024 threads) and many (512), each on its quick and on its general path
(csrc/sampling.cu): the four choose the same tokens, whatever else the call holds."""

import numpy as np
import pytest
import torch

from sleuth_b200.sampling.config import SamplingConfig
from sleuth_b200.sampling.sampler import Sampler
from test_sampling_paths_gpu import DEV, HELD

pytestmark = pytest.mark.gpu
LOWEST = -3.4028234663852886e38


def rows_of(kind, vocab, gen):
    x = torch.randn((6, vocab), generator=gen) * 2.5
    if kind == "narrow":                                  # all weights alike: the steps of the histogram have to be narrow too
        x *= 0.02
    elif kind == "narrow and far":
        x = x * 0.002 + 300.0
    elif kind == "stretches banned":                      # whole warps without an allowed token, by either sign of a ban
        x[:, vocab // 4: vocab // 2] = float("-inf")
        x[:3, vocab // 2: 3 * vocab // 4] = LOWEST
    elif kind == "few allowed":                           # fewer than top-k asks for
        keep = torch.randint(0, vocab, (6, 12), generator=gen)
        x = torch.full_like(x, float("-inf")).scatter(1, keep, x.gather(1, keep))
        x[3:] = x[3:].clamp_min(LOWEST)
    elif kind == "no number":
        x[1, vocab // 3] = float("nan")
        x[2, vocab // 2] = float("inf")
        x[4, 5:] = float("-inf")
    return x


@pytest.mark.parametrize("vocab", [1031, 50257, 151936])
@pytest.mark.parametrize("kind", ["normal", "narrow", "narrow and far", "stretches banned", "few allowed", "no number"])
def test_few_and_many_rows_quick_and_general_path(vocab, kind):
    gen = torch.Generator().manual_seed(vocab + len(kind))
    x = rows_of(kind, vocab, gen)
    wide = torch.full((6, HELD + 8), -1e30)
    wide[:, :vocab] = x
    forms = [(x.to(DEV), vocab), (x.repeat(4, 1).to(DEV), vocab), (wide.to(DEV), HELD + 8), (wide.repeat(4, 1).to(DEV), HELD + 8)]
    samplers = [Sampler(DEV, v) for _, v in forms]
    u = np.random.default_rng(vocab).random((3, 6), dtype=np.float32)
    for k, p, m in [(0, 1.0, 0.0), (0, 1.0, 0.05), (1, 1.0, 0.0), (50, 0.9, 0.0), (400, 0.98, 0.05), (1024, 0.9, 0.0), (1030, 0.9, 0.0), (0, 0.7, 0.0),
                    (0, 0.98, 0.1), (0, 1e-6, 0.0)]:
        for t in (0.3, 0.8, 20.0):
            cfg = SamplingConfig(temperature=t, top_k=k, top_p=p, min_p=m)
            for uu in u:
                got = [s.choose(logits, cfg, np.tile(uu, logits.shape[0] // 6)).cpu().view(-1, 6) for s, (logits, _) in zip(samplers, forms)]
                for other in got:
                    assert (other == got[0][:1]).all(), (k, p, m, t, [g.tolist() for g in got])
