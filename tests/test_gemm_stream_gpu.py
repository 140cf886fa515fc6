"""The weight-streaming tcgen05 product (csrc/gemm_stream.cu) against float64: rows at the edges of its token tiles, features off the 128 (64
gate and 64 up) of a tile and off the four of a store, every number of blocks that share K, and a last slice of K that is not full."""

import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16", "f32", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (16, 200, 520), (17, 131, 1024), (33, 1024, 2048), (64, 66, 576), (65, 640, 1000), (128, 257, 3072)])
def test_product(mode, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn((2 if mode == "swiglu" else 1) * N, K, generator=g) / 16).bfloat16().to(DEV)
    base = torch.randn(M, N, generator=g).to(DEV)
    full = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    # float32 sums of K exact products, then (where the output is bfloat16) one rounding to 8 bits
    bound = 2.0 ** -23 * (K / 16 + 20) * size
    if mode == "swiglu":
        gate, up = full[:, :N], full[:, N:]
        ref = torch.nn.functional.silu(gate) * up
        bound = (1.2 * bound[:, :N] * up.abs() + gate.abs() * bound[:, N:]) + 2.0 ** -20 * ref.abs()
    else:
        ref = full + (base.double() if mode == "add" else 0)
    half = mode in ("bf16", "swiglu")
    bound = bound + (2.0 ** -8 if half else 2.0 ** -22) * ref.abs() + 1e-6
    for splits in range(0, min(8, -(-K // 64)) + 1):
        out = base.clone() if mode == "add" else torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16 if half else torch.float32)
        ops().gemm_stream(x, w, out, mode, static_weight=splits % 2 == 0, splits=splits)
        assert ((out.double() - ref).abs() <= bound).all(), splits
        if splits:
            again = base.clone() if mode == "add" else torch.empty_like(out)
            ops().gemm_stream(x, w, again, mode, splits=splits)
            assert torch.equal(out, again)
    kernel_ops.gemm_tc_check(torch.device(DEV))


def test_other_gates():
    g = torch.Generator().manual_seed(4)
    M, N, K = 40, 200, 512
    x, w = torch.randn(M, K, generator=g).bfloat16().to(DEV), (torch.randn(2 * N, K, generator=g) / 16).bfloat16().to(DEV)
    full = x.double() @ w.double().T
    for gate in (("relu", 0.0, 1.0), ("clamped_swish", 1.5, 1.702), ("gelu_tanh", 0.0, 1.0)):
        out, plain = torch.empty(M, N, device=DEV, dtype=torch.bfloat16), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
        ops().gemm_stream(x, w, out, "swiglu", gate=gate)
        ops().gated_act(full.bfloat16(), plain, gate[0], None, gate[1], gate[2])
        torch.testing.assert_close(out.float(), plain.float(), rtol=3e-2, atol=3e-2)
