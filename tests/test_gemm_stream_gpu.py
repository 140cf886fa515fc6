"""The weight-streaming tcgen05 product (csrc/gemm_stream.cu) against float64: rows at the edges of its token tiles, features off the 128 (64
gate and 64 up) of a tile and off the four of a store, every number of blocks that share K, and a last slice of K that is not full."""

import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16", "f32", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (16, 200, 520), (17, 131, 1024), (33, 1024, 2048), (64, 66, 576), (63, 640, 1000), (48, 257, 3072)])
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


@pytest.mark.parametrize("mode", ["bf16", "f32", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K,offset", [(13, 131, 576, 1), (64, 132, 520, 1), (20, 260, 576, 2), (33, 1027, 1024, 3)])
def test_results_that_lie_off_16_bytes(mode, M, N, K, offset):
    """A result at any element's address, rows of any length: the same bits as in a buffer of its own."""
    g = torch.Generator().manual_seed(N + offset)
    x = torch.randn(M, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn((2 if mode == "swiglu" else 1) * N, K, generator=g) / 16).bfloat16().to(DEV)
    dtype = torch.bfloat16 if mode in ("bf16", "swiglu") else torch.float32
    own = torch.full((M, N), 0.5, device=DEV, dtype=dtype)
    around = torch.full((M * N + offset + 8,), 0.5, device=DEV, dtype=dtype)
    ops().gemm_stream(x, w, own, mode, splits=2)
    ops().gemm_stream(x, w, around[offset:offset + M * N].view(M, N), mode, splits=2)
    assert torch.equal(around[offset:offset + M * N].view(M, N), own)
    assert (around[:offset] == 0.5).all() and (around[offset + M * N:] == 0.5).all()


def test_chunked_step_with_an_odd_vocabulary():
    """A step cut into chunks whose later logits begin at a row off 16 bytes gives the logits of the uncut step."""
    from sleuth_b200.engine.engine import Engine
    vocab = 8209
    cfg = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "vocab_size": vocab, "hidden_size": 1024, "intermediate_size": 256,
           "num_hidden_layers": 1, "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64, "rope_theta": 1e4, "rms_norm_eps": 1e-6,
           "attention_bias": False, "tie_word_embeddings": False, "max_position_embeddings": 256}
    gen = torch.Generator().manual_seed(2)
    prompts = [torch.randint(0, vocab, (50,), generator=gen).tolist() for _ in range(30)]
    logits = []
    for most in (8192, 50 * 13, 50 * 17):
        eng = Engine.from_config(cfg, seed=3, dtype="bf16", max_seq_len=64, max_tokens=30 * 64, max_sequences=32, max_step_tokens=most)
        logits.append(eng.step([(s, p, (len(p) - 1,)) for s, p in zip(eng.open(30), prompts)]).cpu())
    for other in logits[1:]:
        # the layers' products run on other kernels for other numbers of rows: bfloat16 roundings of one layer
        torch.testing.assert_close(other, logits[0], rtol=0, atol=0.03 * float(logits[0].abs().max()))
