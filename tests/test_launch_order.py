"""What kernels may do before the kernel in front has finished, and when they let the next one begin, without a GPU: only a matrix
that no kernel writes is read early, and the next kernel starts after a block has its tensor memory."""

import re

import torch

from sleuth_b200.kernels import library, ops
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


def test_the_next_kernel_starts_only_when_tensor_memory_is_taken():
    """A block that lets the next kernel begin before it has its own tensor memory may find it taken by a block that waits for this
    one's grid: neither could go on. So between the allocation and the signal lies a barrier of the block, and a warp that has only
    arrived at it (and may be ahead of the allocation) does not signal."""
    seen = 0
    for path in sorted(library.CSRC.glob("*.cu")):
        text = path.read_text()
        for kernel in re.split(r"\n(?=(?:template <[^\n]*>\n)?__global__)", text)[1:]:
            allocated, signal = kernel.find("tcgen05.alloc"), kernel.find("pdl_launch_dependents()")
            if allocated < 0 or signal < 0:
                continue
            between = kernel[allocated:signal]
            assert re.search(r"__syncthreads\(\)|cluster_sync_all\(\)|bar\.sync", between), path.name
            line = kernel[kernel.rfind("\n", 0, signal) + 1:signal]
            assert "bar.arrive" not in kernel[:signal] or "if (" in line, path.name
            seen += 1
    assert seen >= 5
