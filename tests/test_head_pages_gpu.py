"""Whole prompts of heads with a rotated key part or values of another width on the tcgen05 attention (csrc/head_pages.cu): rows as
they are laid out, the attention through them against the kernel for heads as they are, and the gates."""

import numpy as np
import pytest
import torch

from sleuth_b200.kernels import ops as kernel_ops
from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


# Rows of 64 and 128; a rotated part that is not all turned, none at all; values as wide as the row and narrower; sequences of one
# token, of whole pages, of one token more; windows.
@pytest.mark.parametrize("H,dn,P,rot,dv", [(3, 64, 32, 32, 64), (5, 24, 8, 8, 48), (2, 96, 32, 16, 128), (4, 40, 0, 0, 16), (2, 32, 32, 32, 8)])
@pytest.mark.parametrize("window", [0, 100])
def test_rows_and_attention(H, dn, P, rot, dv, window):
    o, dt = ops(), torch.bfloat16
    counts, W, scale = [1, 65, 300, 64, 128], 64 if max(dn + P, dv) <= 64 else 128, 0.2
    T, n = sum(counts), len(counts)
    g = torch.Generator().manual_seed(H + dn)
    rand = lambda *shape: torch.randn(*shape, generator=g).to(dt).to(DEV)
    q, kv, k_rot = rand(T, H, dn + P), rand(T, H * (dn + dv)), rand(T, P)
    angles = torch.outer(torch.arange(max(counts), dtype=torch.float32), 1000.0 ** (-torch.arange(max(rot // 2, 1), dtype=torch.float32) / max(rot // 2, 1)))
    cos, sin = (angles.cos().to(DEV), angles.sin().to(DEV)) if rot else (None, None)
    starts = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    i32 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32)).to(DEV)
    seq_of, pos_of = np.repeat(np.arange(n), counts), np.concatenate([np.arange(c) for c in counts])
    pages = kernel_ops.prompt_pages(T, n)
    k_pages, v_pages = torch.full((pages, H, 64, W), float("nan"), dtype=dt, device=DEV), torch.zeros(pages, H, 64, W, dtype=dt, device=DEV)
    rows = torch.full((T, H, W), float("nan"), dtype=dt, device=DEV)
    o.head_pages(q, kv, k_rot, rows, k_pages, v_pages, cos, sin, i32(seq_of), i32(pos_of), i32(starts), dn, dv, rot)
    first = starts[:-1] // 64 + np.arange(n)
    at = torch.as_tensor(first[seq_of] + pos_of // 64).to(DEV), torch.as_tensor(pos_of % 64).to(DEV)
    keys, values = k_pages.permute(0, 2, 1, 3)[at], v_pages.permute(0, 2, 1, 3)[at]
    want = torch.zeros(T, H, W, dtype=dt, device=DEV)
    want[..., :dn], want[..., dn:dn + P] = kv[:, :H * dn].view(T, H, dn), k_rot[:, None]
    assert torch.equal(keys, want)
    want = torch.zeros(T, H, W, dtype=dt, device=DEV)
    want[..., :dv] = kv[:, H * dn:].view(T, H, dv)
    assert torch.equal(values, want)
    turned = q.float()
    if rot:
        c, s = (f[torch.as_tensor(pos_of).to(DEV)][:, None] for f in (cos, sin))
        a, b = q[..., dn:dn + rot // 2].float(), q[..., dn + rot // 2:dn + rot].float()
        turned[..., dn:dn + rot] = torch.cat([a * c - b * s, b * c + a * s], -1)
    torch.testing.assert_close(rows[..., :dn + P].float(), turned, rtol=2 ** -7, atol=1e-5)
    assert not rows[..., dn + P:].any()

    table = np.zeros((n, 5), dtype=np.int32)
    for i, c in enumerate(counts):
        table[i, :-(-c // 64)] = first[i] + np.arange(-(-c // 64))
    y = torch.full((T, H, W), float("nan"), dtype=dt, device=DEV)
    o.attention_tc(rows, k_pages, v_pages, y.view(T, H * W), i32(starts), i32([0] * n), i32(counts), i32(table), max(counts), H, H, W, window, scale,
                   max_keys=max(counts))
    at = 0
    for i, c in enumerate(counts):
        qq, kk, vv = (x[at:at + c].double() for x in (rows, keys, values))
        s = torch.einsum("ihd,jhd->hij", qq, kk) * scale
        p = torch.arange(c, device=DEV)
        hidden = (p[None, :] > p[:, None]) | ((p[None, :] <= p[:, None] - window) if window else False)
        ref = torch.einsum("hij,jhd->ihd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), vv)
        torch.testing.assert_close(y[at:at + c].double(), ref, rtol=2e-2, atol=2e-2)
        at += c

    gate, head_gate = rand(T, H * dv), torch.randn(T, H + 3, generator=g).to(DEV)[:, 1:H + 1]
    cut = y[..., :dv].reshape(T, H * dv)
    for kw, z in (({}, None), ({"gate": gate}, gate.double()), ({"head_gate": head_gate}, head_gate.double().repeat_interleave(dv, 1))):
        out = torch.full((T, H * dv), float("nan"), dtype=dt, device=DEV)
        o.head_rows(y, out, **kw)
        ref = cut.double() * (torch.sigmoid(z) if z is not None else 1.0)
        torch.testing.assert_close(out.double(), ref, rtol=2 ** -7, atol=1e-6)
