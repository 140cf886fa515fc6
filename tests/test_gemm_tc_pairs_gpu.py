"""Products from 512 rows on with large matrices go to pairs of blocks: rows and features off their tiles, every epilogue."""

import pytest
import torch

from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16", "f32", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(511, 2560, 4096), (512, 2560, 4096), (700, 2600, 4104), (1030, 4097, 2560)])
def test_product(mode, M, N, K):
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn((2 if mode == "swiglu" else 1) * N, K, generator=g) / 64).bfloat16().to(DEV)
    base = torch.randn(M, N, generator=g).to(DEV)
    full = x.double() @ w.double().T
    ref = torch.nn.functional.silu(full[:, :N]) * full[:, N:] if mode == "swiglu" else full + (base.double() if mode == "add" else 0)
    half = mode in ("bf16", "swiglu")
    out = base.clone() if mode == "add" else torch.empty(M, N, device=DEV, dtype=torch.bfloat16 if half else torch.float32)
    ops().gemm_tc(x, w, out, mode)
    torch.testing.assert_close(out.double(), ref, rtol=1e-2 if half else 1e-4, atol=1e-2 if half else 1e-3)
