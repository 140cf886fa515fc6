"""Single-token attention of batches that fill the GPU several times over (csrc/attention_flash.cu, attn_decode_kernel with three
page buffers and with two), post-processed queries and the fused form, against float64: positions around the edges of a warp's keys
and of pages and several hundred keys (the ring of buffers goes round many times), windows and chunks that begin anywhere in a page."""

import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, make_cache, ops

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
POSITIONS = [0, 1, 15, 16, 30, 31, 32, 33, 47, 48, 62, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 223, 300, 415, 416, 447, 511, 640, 702, 703]


def first_key(pos, window):
    return max(0, pos - window + 1) if window > 0 else (pos // -window * -window if window < 0 else 0)


def batch(n):
    return [(POSITIONS[i % len(POSITIONS)] + (37 * (i // len(POSITIONS)))) for i in range(n)]


def reference(q, ks, vs, pasts, window, scale):
    """q [n, H, hd]; ks, vs per sequence [pos + 1, K, hd]."""
    out = []
    for i, pos in enumerate(pasts):
        lo, rep = first_key(pos, window), q.shape[1] // ks[i].shape[1]
        k, v = (t[lo:pos + 1].double().repeat_interleave(rep, 1) for t in (ks[i], vs[i]))
        p = torch.softmax(torch.einsum("hd,jhd->hj", q[i].double(), k) * scale, 1)
        out.append(torch.einsum("hj,jhd->hd", p, v))
    return torch.stack(out)


d = lambda a: None if a is None else torch.as_tensor(a).to(DEV)
ints = lambda a: d(np.asarray(a, dtype=np.int32))


# 64 x 8, 75 x 6 and 460 x 1 blocks of one slice: three page buffers; (160 sequences of 40 heads, 2 kv heads): two tiles of query rows, 2 x 2 x 160 blocks, two
@pytest.mark.parametrize("n,heads,kv_heads", [(64, 16, 8), (75, 24, 6), (460, 3, 1), (160, 40, 2)])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [0, 45, 100, 77, 200, -48, -96])
def test_post_processed_queries(n, heads, kv_heads, hd, window):
    gen = torch.Generator().manual_seed(n + hd + window)
    pasts, scale = batch(n), 1.0 / math.sqrt(hd)
    k_pool, v_pool, table, ks, vs = make_cache([p + 1 for p in pasts], kv_heads, hd, BF, gen)
    q = torch.randn(n, heads, hd, generator=gen).to(BF)
    out = torch.full((n, heads * hd), float("nan"), dtype=BF, device=DEV)
    ops().attention_decode(d(q), d(k_pool), d(v_pool), out, ints(range(n + 1)), ints(pasts), d(table), heads, kv_heads, hd, window, scale, 1, None)
    torch.testing.assert_close(out.cpu().double().view(n, heads, hd), reference(q, ks, vs, pasts, window, scale), rtol=2e-2, atol=1.5e-2)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [0, 100, 77, -96])
@pytest.mark.parametrize("n", [64, 80])      # three page buffers; two at heads of 128
def test_fused_form(n, hd, window):
    heads, kv_heads, eps = 16, 8, 1e-5
    gen = torch.Generator().manual_seed(hd + window)
    pasts, scale, rows = batch(n), 1.0 / math.sqrt(hd), heads + 2 * kv_heads
    k_pool, v_pool, table, ks, vs = make_cache([p + 1 for p in pasts], kv_heads, hd, BF, gen)
    qkv, bias = torch.randn(n, rows * hd, generator=gen).to(BF), torch.randn(rows * hd, generator=gen) * 0.1
    qg, kg = 1 + 0.1 * torch.randn(hd, generator=gen), 1 + 0.1 * torch.randn(hd, generator=gen)
    ang = torch.outer(torch.arange(1100, dtype=torch.float32), 1.0 / (1e4 ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd)))
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    x = qkv.double().view(n, rows, hd) + bias.double().view(rows, hd)

    def post(v, gain):
        v = v * torch.rsqrt((v * v).mean(-1, keepdim=True) + eps) * gain.double()
        c, s = cos[pasts].double()[:, None, :], sin[pasts].double()[:, None, :]
        a, b = v[..., :hd // 2], v[..., hd // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1).to(BF)

    q, k_new, v_new = post(x[:, :heads], qg), post(x[:, heads:heads + kv_heads], kg), x[:, heads + kv_heads:].to(BF)
    for i, p in enumerate(pasts):                # the pools' newest rows hold something else
        ks[i][p], vs[i][p] = k_new[i], v_new[i]
    kp, vp, out = d(k_pool), d(v_pool), torch.full((n, heads * hd), float("nan"), dtype=BF, device=DEV)
    ops().attention_decode(None, kp, vp, out, ints(range(n + 1)), ints(pasts), d(table), heads, kv_heads, hd, window, scale, 1, None, qkv=d(qkv),
                           qkv_kv_heads=kv_heads, bias=d(bias), q_gain=d(qg), k_gain=d(kg), cos=d(cos), sin=d(sin), eps=eps)
    torch.testing.assert_close(out.cpu().double().view(n, heads, hd), reference(q, ks, vs, pasts, window, scale), rtol=2e-2, atol=1.5e-2)
    page = torch.tensor([int(table[i, p // 64]) for i, p in enumerate(pasts)])
    row = torch.tensor(pasts) % 64
    want_k, want_v = k_pool.clone(), v_pool.clone()
    want_k[page, :, row], want_v[page, :, row] = k_new, v_new
    for got, want in ((kp.cpu(), want_k), (vp.cpu(), want_v)):      # the appended rows, and no other row of the cache
        torch.testing.assert_close(got[page, :, row].float(), want[page, :, row].float(), rtol=2e-2, atol=2e-2)
        got[page, :, row] = want[page, :, row]
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [0, 77, -96])
def test_a_sequences_bits_do_not_depend_on_the_batch(hd, window):
    """Any number of sequences beside it, three page buffers or two: the same bits for a sequence."""
    n, heads, kv_heads = 80, 16, 8
    gen = torch.Generator().manual_seed(hd + window)
    pasts, scale = batch(n), 1.0 / math.sqrt(hd)
    k_pool, v_pool, table, _, _ = make_cache([p + 1 for p in pasts], kv_heads, hd, BF, gen)
    k_pool, v_pool, table, q = d(k_pool), d(v_pool), d(table), d(torch.randn(n, heads, hd, generator=gen).to(BF))

    def run(a, b):
        out = torch.full((b - a, heads * hd), float("nan"), dtype=BF, device=DEV)
        ops().attention_decode(q[a:b].contiguous(), k_pool, v_pool, out, ints(range(b - a + 1)), ints(pasts[a:b]), table[a:b].contiguous(), heads, kv_heads, hd,
                               window, scale, 1, None)
        return out

    together = run(0, n)
    for a, b in ((0, 16), (16, 32), (20, 60), (15, 79), (63, 64)):
        assert torch.equal(run(a, b), together[a:b])
