"""The 32-bit product on the tensor cores (csrc/gemm_f32_tc.cu): every form against float64 with a bound that follows from its order of
sums, the same bits whatever the form and the rows beside a row, and operands that are infinite, NaN, huge and tiny."""

import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu

FORMS = [(128, 1, 16), (64, 1, 16), (32, 1, 8)] + [(16, 1, 8)] + [(16, s, 16) for s in (2, 4, 8)] + [(32, s, 16) for s in (1, 2, 4, 8)]


def bound_of(a, w, K):
    """In units of 2^-24 of the products' absolute sum: 2 for the partial products that are left out (2^-8 x 2^-16, twice); a chunk of 64
    ends with four additions at full size, each with sixteen products aligned to the largest and the sum truncated (4 x 4), after twenty
    at 2^-7 of it (1); then one rounding a chunk."""
    steps = 2.0 + 16.0 + 1.0 + K / 64
    return 2.0 ** -24 * steps * (a.double().abs() @ w.double().abs().T)


# Tiles of 128 features with a ragged last one, rows at the edges of every tile, a last chunk of 4 to 60 values, one chunk more than the
# blocks of a cluster share evenly, fewer chunks than blocks, sums that fit shared memory for fewer rows than a tile has tokens.
@pytest.mark.parametrize("M,N,K", [(1, 512, 1024), (15, 520, 1028), (16, 1000, 2108), (17, 640, 260), (33, 4100, 300), (64, 1024, 3072),
                                   (65, 513, 1092), (129, 1030, 1024), (300, 2050, 516), (7, 512, 4096)])
def test_every_form_gives_the_same_bits(M, N, K):
    g = torch.Generator().manual_seed(M * 7 + N + K)
    a, w, bias = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    want = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a, w, want, form=(128, 1, 16))
    ref = a.double() @ w.double().T
    assert ((want.double() - ref).abs() <= bound_of(a, w, K)).all()
    for form in FORMS + [(0, 0, 0)]:
        out = torch.full((M, N), float("nan"), device=DEV)
        try:
            ops().gemm_f32(a, w, out, form=form, static_weight=True)
        except RuntimeError as e:
            assert "do not fit" in str(e) and form[0] == 16 and form[1] < 8 and K > 2000, form      # never the rule's choice
            continue
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
    ops().gemm_f32(shifted, w, out, form=(64, 1, 16))
    assert torch.equal(out, want)
    kernel_ops.gemm_tc_check(torch.device(DEV))


@pytest.mark.parametrize("M,N,K", [(1, 256, 1024), (16, 300, 1028), (33, 2050, 300), (65, 257, 1092), (300, 1000, 516)])
@pytest.mark.parametrize("gate", [None, ("clamped_swish", 1.5, 1.702), ("gelu_tanh", 0.0, 1.0)])
def test_gated_product_is_product_and_activation(M, N, K, gate):
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g), torch.randn(2 * N, K, generator=g) / 16
    a[M // 2, 3] = float("inf")
    a, w = a.to(DEV), w.to(DEV)
    both, want = torch.empty(M, 2 * N, device=DEV), torch.empty(M, N, device=DEV)
    ops().gemm_f32(a, w, both, form=(0, 0, 0))
    ops().gated_act(both, want, gate[0] if gate else "silu", None, *(gate[1:] if gate else (0.0, 1.0)))
    for form in [f for f in FORMS if f[0] <= 32] + [(0, 0, 0)]:
        out = torch.full((M, N), 7.0, device=DEV)
        ops().gemm_f32_gated(a, w, out, gate, form=form)
        assert torch.equal(out.nan_to_num(5.0, 6.0, -6.0), want.nan_to_num(5.0, 6.0, -6.0)), form
    kernel_ops.gemm_tc_check(torch.device(DEV))


@pytest.mark.parametrize("N,K", [(1024, 1024), (1024, 3072), (4096, 2560)])
def test_error_is_no_larger_than_the_fma_kernels(N, K):
    g = torch.Generator().manual_seed(N + K)
    a, w = torch.randn(200, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) * 0.02).to(DEV)
    ref = a.double() @ w.double().T
    tensor, fma = torch.empty(200, N, device=DEV), torch.empty(200, N, device=DEV)
    ops().gemm_f32(a, w, tensor, form=(0, 0, 0))
    kernel_ops.lib().call("slb_gemm_f32", a.data_ptr(), w.data_ptr(), None, fma.data_ptr(), 200, N, K, K, K, N, 0, 0, kernel_ops.current_stream())
    error = lambda x: float((x.double() - ref).norm())
    assert error(tensor) <= error(fma)


@pytest.mark.parametrize("form", [(16, 1, 8), (128, 1, 16), (16, 4, 16), (32, 2, 16)])
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
    assert ((out.double() - ref).abs()[finite] <= bound_of(a, w, K).nan_to_num()[finite] + 1e-40).all()
    assert out[9, 7] == float("inf") and torch.isnan(out[3]).all()
    for m, n in ((1, 5), (1, 100), (2, 200), (10, 4), (1, 4), (5, 4)):
        want = torch.tensor(0.0)
        for k in range(K):
            want = want + a[m, k] * w[n, k]
        assert torch.equal(torch.isnan(out[m, n]), torch.isnan(want)) and (torch.isnan(want) or out[m, n] == want), (m, n)
