"""What the products hand their kernels about the order of launches, without a GPU: only a matrix that no kernel writes may be
read before the kernel in front has finished."""

import torch

from sleuth_b200.kernels import ops
from sleuth_b200.parts.linear import Linear


def test_only_loaded_matrices_are_read_early(monkeypatch):
    calls = []
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "lib", lambda: type("Lib", (), {"call": lambda self, name, *a: calls.append((name, a))})())
    a, w, out = torch.zeros(3, 8), torch.zeros(5, 8), torch.zeros(3, 5)
    ops.gemm_f32(a, w, out, stream=0)
    ops.gemm_f32(a, w, out, accumulate=True, stream=0)
    Linear(w, torch.float32).forward(a, out=out, stream=0)
    Linear(w, torch.float32).forward(a, into=out, stream=0)
    assert [c[0] for c in calls] == ["slb_gemm_f32"] * 4
    assert [c[1][10:12] for c in calls] == [(0, 0), (1, 0), (0, 1), (1, 1)]      # accumulate, static weight
