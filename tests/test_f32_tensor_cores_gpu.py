"""The 32-bit product on the tensor cores (csrc/gemm_f32_tc.cu): every form against float64 with a bound that follows from its order of
sums, the same bits whatever the form and the rows beside a row, and operands that are infinite, NaN, huge and tiny."""

import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu

FORMS = [0, 1, 32, 64, 128]      # 1: on mma.sync, tiles of 8, 16 and 32 rows; the others on tcgen05, by tokens of a tile


def bound_of(a, w, K):
    """In units of 2^-24 of the products' absolute sum: 2 for the partial products that are left out (2^-8 x 2^-16, twice); a chain of 32
    ends with two additions at full size, each with sixteen products aligned to the largest and the sum truncated (2 x 4), after ten
    at 2^-7 of it (1); then the two chains, two chunks, and one rounding a pair of chunks."""
    steps = 2.0 + 8.0 + 1.0 + 2.0 + K / 128
    return 2.0 ** -24 * steps * (a.double().abs() @ w.double().abs().T)


# Tiles of 128 and 16 features with a ragged last one, rows at the edges of every tile, a last chunk of 4 to 60 values, odd numbers of chunks, fewer
# than the few-rows kernel has warps and one more than they share evenly, several of its tiles a block, both of its block sizes.
@pytest.mark.parametrize("M,N,K", [(1, 512, 1024), (8, 5000, 1088), (9, 4741, 1024), (15, 520, 1028), (16, 1000, 2108), (17, 640, 260), (32, 2369, 4), (33, 4100, 300),
                                   (64, 1024, 3072), (65, 513, 1092), (129, 1030, 1024), (300, 2050, 516), (7, 512, 4096), (40, 4800, 68)])
def test_every_form_gives_the_same_bits(M, N, K):
    g = torch.Generator().manual_seed(M * 7 + N + K)
    a, w, bias = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    want = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a, w, want, form=128)
    ref = a.double() @ w.double().T
    assert ((want.double() - ref).abs() <= bound_of(a, w, K)).all()
    for form in FORMS:
        out = torch.full((M, N), float("nan"), device=DEV)
        ops().gemm_f32(a, w, out, form=form, static_weight=True)
        assert torch.equal(out, want), form
        ops().gemm_f32(a, w, out, accumulate=True, form=form)
        assert torch.equal(out, want + want), form
        ops().gemm_f32(a, w, out, bias, form=form)
        assert torch.equal(out, want + bias), form
        for rows in (1, 5, 40):
            if rows < M:
                some = torch.empty(rows, N, device=DEV)
                ops().gemm_f32(a[M - rows:].contiguous(), w, some, form=form)
                assert torch.equal(some, want[M - rows:]), form
    shifted = torch.empty(M * K + 1, device=DEV)[1:].view(M, K).copy_(a)      # no 16-byte reads
    out = torch.empty(M, N, device=DEV)
    for form in (1, 64):
        ops().gemm_f32(shifted, w, out, form=form)
        assert torch.equal(out, want)
    kernel_ops.gemm_tc_check(torch.device(DEV))


@pytest.mark.parametrize("M,N,K", [(1, 256, 1024), (8, 2500, 1028), (16, 300, 1028), (32, 2401, 520), (33, 2050, 300), (64, 257, 1092)])
@pytest.mark.parametrize("gate", [None, ("clamped_swish", 1.5, 1.702), ("gelu_tanh", 0.0, 1.0)])
def test_gated_product_is_product_and_activation(M, N, K, gate):
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g), torch.randn(2 * N, K, generator=g) / 16
    a[M // 2, 3] = float("inf")
    a, w = a.to(DEV), w.to(DEV)
    both, want = torch.empty(M, 2 * N, device=DEV), torch.empty(M, N, device=DEV)
    ops().gemm_f32(a, w, both, form=0)
    ops().gated_act(both, want, gate[0] if gate else "silu", None, *(gate[1:] if gate else (0.0, 1.0)))
    for static in (False, True):
        out = torch.full((M, N), 7.0, device=DEV)
        ops().gemm_f32_gated(a, w, out, gate, static_weight=static)
        assert torch.equal(out.nan_to_num(5.0, 6.0, -6.0), want.nan_to_num(5.0, 6.0, -6.0))
    kernel_ops.gemm_tc_check(torch.device(DEV))


@pytest.mark.parametrize("N,K", [(1024, 1024), (1024, 2048), (1024, 3072), (4096, 2560), (512, 4100)])
@pytest.mark.parametrize("values", ["normal", "one sign", "uniform", "narrow", "shifted", "wide"])
def test_error_is_no_larger_than_the_fma_kernels(N, K, values):
    """Over the matrices that the rule sends to the tensor cores, for operands of mean zero and of one sign (where a truncated sum is a
    bias), of little spread and of much."""
    g = torch.Generator().manual_seed(N + K)
    a, w = torch.randn(200, K, generator=g), torch.randn(N, K, generator=g) * 0.02
    if values == "one sign":
        a, w = a.abs(), w.abs()
    elif values in ("uniform", "narrow"):
        a, w = torch.rand(200, K, generator=g) + (values == "narrow"), torch.rand(N, K, generator=g) + (values == "narrow")
    elif values == "shifted":
        a, w = a.abs(), w + 0.01
    elif values == "wide":
        a, w = torch.exp(2 * a), torch.exp(100 * w)
    a, w = a.to(DEV), w.to(DEV)
    assert kernel_ops.f32_on_tensor_cores(N, K, w.data_ptr())
    ref = a.double() @ w.double().T
    tensor, fma = torch.empty(200, N, device=DEV), torch.empty(200, N, device=DEV)
    ops().gemm_f32(a, w, tensor, form=0)
    ops().gemm_f32(a, w, fma, form="fma")
    error = lambda x: float((x.double() - ref).norm())
    assert error(tensor) <= error(fma)


@pytest.mark.parametrize("form", [1, 32, 64, 128])
@pytest.mark.parametrize("size,other", [(1e-33, 1.0), (1e-36, 1e28), (1e-40, 1e30), (1e-43, 1e20), (1e-36, 1e36), (3e-39, 3e-2)])
def test_tiny_values_lose_nothing(form, size, other):
    """Values whose low parts lie below the smallest bfloat16, subnormal ones too, in either operand, beside others that bring the
    result back to ordinary size (or not: then it rounds to a multiple of 2^-149)."""
    M, N, K = 20, 520, 1024
    g = torch.Generator().manual_seed(5)
    for tiny_weights in (False, True):
        a, w = torch.randn(M, K, generator=g) * (other if tiny_weights else size), torch.randn(N, K, generator=g) * (size if tiny_weights else other)
        a, w = a.to(DEV), w.to(DEV)
        out = torch.full((M, N), float("nan"), device=DEV)
        ops().gemm_f32(a, w, out, form=form)
        # (where a sum is formed again by FMA: chains of an eighth of K)
        bound = torch.maximum(bound_of(a, w, K), 2.0 ** -24 * (K / 8 + 8) * (a.double().abs() @ w.double().abs().T) * (other > 1e31))
        assert ((out.double() - a.double() @ w.double().T).abs() <= bound + 2.0 ** -148).all()


@pytest.mark.parametrize("form", [1, 32, 64, 128])
def test_values_at_the_ends_of_the_range(form):
    M, N, K = 20, 520, 512
    g = torch.Generator().manual_seed(11)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    a[1, 5], a[2, 7], a[3, 9], a[3, 10] = float("inf"), float("-inf"), float("nan"), float("inf")
    w[4, 11] = float("inf")
    a[5], w[6] = 0.0, 0.0
    a[5, 3], w[6, 3] = 3.4e38, 1.0              # rounds beyond the largest bfloat16; the product itself is finite
    a[7] *= 1e30
    a[8] *= 1e-30
    a[9], a[9, 300] = 0.0, 3.4e38
    w[7, 300] = 2.0                             # 6.8e38: infinite in float32
    out = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a.to(DEV), w.to(DEV), out, form=form)
    out = out.cpu()
    # what each product and sum gives in float32
    ref = (a.double().to(DEV) @ w.double().to(DEV).T).cpu()
    finite = torch.isfinite(a).all(1)[:, None] & torch.isfinite(w).all(1)[None, :] & (ref.abs() < 3.4e38)
    # (row 7: beyond 2^80, formed by FMA in chains of 128)
    bound = bound_of(a, w, K).nan_to_num()
    bound[7] = torch.maximum(bound[7], 2.0 ** -24 * (128 + 8) * (a[7].double().abs() @ w.double().abs().T).nan_to_num())
    assert ((out.double() - ref).abs()[finite] <= bound[finite] + 1e-40).all()
    assert out[9, 7] == float("inf") and torch.isnan(out[3]).all()
    for m, n in ((1, 5), (1, 100), (2, 200), (10, 4), (1, 4), (5, 4)):
        want = torch.tensor(0.0)
        for k in range(K):
            want = want + a[m, k] * w[n, k]
        assert torch.equal(torch.isnan(out[m, n]), torch.isnan(want)) and (torch.isnan(want) or out[m, n] == want), (m, n)
