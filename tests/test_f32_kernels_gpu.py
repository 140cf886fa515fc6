"""The true 32-bit kernels (csrc/gemm_f32.cu, csrc/attention_f32.cu) at the edges of their tiles, against float64, and their
promise that a row's bits depend neither on the rows beside it nor on how a sequence was cut into steps."""

import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import DEV, make_cache, ops, plain_attention

pytestmark = pytest.mark.gpu


# Few rows: tiles of 1, 2, 8, 16, 32 and 64 rows by 8 features (16 from 2,048 features on, 32 from 4,096), segments of 128 and more, a last
# segment that is short or missing, inner dimensions that no 16-byte copy takes. Many rows: tiles of 128 and 96 rows.
@pytest.mark.parametrize("M,N,K", [(1, 8, 4), (1, 9, 132), (2, 8200, 96), (3, 17, 1028), (7, 8192, 260), (8, 1000, 1024), (9, 8195, 644),
                                   (16, 40, 3072), (20, 8200, 132), (33, 100, 1100), (64, 8197, 200), (65, 8, 2052), (100, 24, 77),
                                   (129, 1024, 1024), (700, 1000, 388), (1500, 1030, 64), (1500, 2304, 100), (1100, 6150, 36)])
def test_gemm_f32_error_and_rows(M, N, K):
    g = torch.Generator().manual_seed(M * 7 + N)
    a, w, bias = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    ops().gemm_f32(a, w, out, bias, form="fma")
    ref = a.double() @ w.double().T + bias.double()
    # chains of half a segment, then the halves, at most eight segments and the bias: each step rounds by 2^-24 at most
    seg = max(128, -(-K // 512) * 64)
    steps = min(K, seg) / 2 + 10
    bound = 2.0 ** -24 * steps * 1.01 * (a.double().abs() @ w.double().abs().T + bias.double().abs())
    assert ((out.double() - ref).abs() <= bound).all()
    for rows in (1, 2, 5, 12, 30, 60):
        if rows < M:
            some = torch.empty(rows, N, device=DEV)
            ops().gemm_f32(a[M - rows:].contiguous(), w, some, bias, form="fma")
            assert torch.equal(some, out[M - rows:])
    acc = torch.full((M, N), 2.0, device=DEV)
    ops().gemm_f32(a, w, acc, accumulate=True, form="fma")
    plain = torch.empty(M, N, device=DEV)
    ops().gemm_f32(a, w, plain, form="fma")
    assert torch.equal(acc, plain + 2.0)


# 16- and 32-feature tiles of every row tile with several segments and several tiles a block; inner dimensions of one to seven
# segments, of one and two with tiles side by side in a block (up to eight and four, a last share that is not full), also off a multiple
# of 4; tiles of 128, 96 and 64 rows with one segment and with several; many rows off a multiple of 4.
@pytest.mark.parametrize("M,N,K", [(4, 4100, 1028), (3, 2050, 2052), (8, 2100, 1100), (16, 3000, 1028), (32, 2056, 2052), (1, 5003, 1032), (2, 2051, 516),
                                   (5, 4100, 77), (64, 700, 130), (3, 33, 200), (20, 5000, 300), (60, 12291, 96), (1, 20011, 128), (12, 9001, 388), (64, 4099, 260),
                                   (9, 700, 900), (300, 520, 1030), (1000, 1030, 77), (130, 6150, 333), (700, 300, 129), (2000, 700, 48), (450, 2050, 130), (600, 503, 160),
                                   (300, 1030, 260), (128, 6144, 96), (48, 32801, 160), (7, 40001, 200), (2, 33000, 130), (16, 70001, 68), (1200, 6150, 260), (1500, 1030, 516)])
def test_gemm_f32_groups_of_tiles_and_odd_inner_dimensions(M, N, K):
    test_gemm_f32_error_and_rows(M, N, K)


def run_f32(q, k_pool, v_pool, table, pasts, counts, heads, kv_heads, hd, window, sinks=None):
    o = ops()
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32)).to(DEV)
    out = torch.full((q.shape[0], heads * hd), float("nan"), device=DEV)
    starts = np.concatenate([[0], np.cumsum(counts)])
    floats = o.attention_f32_scratch_floats(len(counts), heads, hd, table.shape[1])
    scratch = torch.full((floats,), float("nan"), device=DEV) if max(counts) == 1 else None
    o.attention_f32(q, k_pool, v_pool, out, d(starts), d(pasts), d(counts), table, max(counts), heads, kv_heads, hd, window,
                    1.0 / math.sqrt(hd), scratch, sinks=sinks)
    return out


@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 2, 128), (5, 1, 64), (8, 8, 64), (16, 1, 128), (3, 3, 128), (12, 2, 64)])
@pytest.mark.parametrize("window,sink", [(0, False), (0, True), (50, False), (200, True), (-96, False)])
def test_attention_f32(heads, kv_heads, hd, window, sink):
    pasts, counts = [0, 70, 0, 129, 300], [1, 1, 200, 64, 130]
    gen = torch.Generator().manual_seed(heads + hd + window)
    lens = [p + c for p, c in zip(pasts, counts)]
    k_pool, v_pool, table, ks, vs = make_cache(lens, kv_heads, hd, torch.float32, gen)
    k_pool, v_pool, table = k_pool.to(DEV), v_pool.to(DEV), table.to(DEV)
    q = torch.randn(sum(counts), heads, hd, generator=gen)
    sinks = torch.randn(heads, generator=gen) if sink else None
    dev_sinks = sinks.to(DEV) if sink else None
    got = run_f32(q.to(DEV), k_pool, v_pool, table, pasts, counts, heads, kv_heads, hd, window, dev_sinks)
    at = 0
    for i, (p, c) in enumerate(zip(pasts, counts)):
        for t in range(c):
            pos = p + t
            lo = max(0, pos - window + 1) if window > 0 else (pos // -window * -window if window < 0 else 0)
            if t % 37 and t not in (0, c - 1):
                continue
            kk = ks[i][lo:pos + 1].double().repeat_interleave(heads // kv_heads, 1)
            vv = vs[i][lo:pos + 1].double().repeat_interleave(heads // kv_heads, 1)
            s = torch.einsum("hd,jhd->hj", q[at + t].double(), kk) / math.sqrt(hd)
            if sink:
                s = torch.cat([s, sinks.double()[:, None]], 1)
            ref = torch.einsum("hj,jhd->hd", torch.softmax(s, 1)[:, :kk.shape[0]], vv)
            # scores to about 1e-6 (chains of 64 at most, values of a few units), weights and sums to a few 1e-6
            torch.testing.assert_close(got[at + t].cpu().double().view(heads, hd), ref, rtol=1e-5, atol=5e-6)
        at += c
    # one sequence at a time, in portions, and its last tokens one by one (all sequences in one step): the same bits
    at = 0
    for i, (p, c) in enumerate(zip(pasts, counts)):
        cuts = [0] + [x for x in (1, 40, 104) if x < c] + [c]
        for x, y in zip(cuts[:-1], cuts[1:]):
            part = run_f32(q[at + x:at + y].to(DEV), k_pool, v_pool, table[i:i + 1], [p + x], [y - x], heads, kv_heads, hd, window, dev_sinks)
            assert torch.equal(part, got[at + x:at + y])
        at += c
    starts = np.concatenate([[0], np.cumsum(counts)])
    for back in (1, 2):
        which = [max(starts[i + 1] - back, starts[i]) for i in range(len(counts))]
        alone = run_f32(q[which].contiguous().to(DEV), k_pool, v_pool, table, [p + int(w - s) for p, w, s in zip(pasts, which, starts)],
                        [1] * len(counts), heads, kv_heads, hd, window, dev_sinks)
        assert torch.equal(alone, got[which])


def test_attention_f32_leaves_later_tokens_out():
    """Infinite values of tokens that a query does not see do not reach it; a NaN key that it sees does."""
    heads, kv_heads, hd, n = 4, 2, 128, 150
    gen = torch.Generator().manual_seed(3)
    k_pool, v_pool, table, ks, vs = make_cache([n], kv_heads, hd, torch.float32, gen)
    q = torch.randn(n, heads, hd, generator=gen).to(DEV)
    clean = run_f32(q, k_pool.to(DEV), v_pool.to(DEV), table.to(DEV), [0], [n], heads, kv_heads, hd, 0)
    v_pool[int(table[0, 1]), :, 36] = float("inf")          # position 100
    k_pool[int(table[0, 1]), :, 46, 0] = float("nan")       # position 110
    got = run_f32(q, k_pool.to(DEV), v_pool.to(DEV), table.to(DEV), [0], [n], heads, kv_heads, hd, 0)
    assert torch.equal(got[:100], clean[:100])
    assert not torch.isfinite(got[100:]).any() and torch.isnan(got[110:]).all()
    one = run_f32(q[120:121], k_pool.to(DEV), v_pool.to(DEV), table.to(DEV), [120], [1], heads, kv_heads, hd, 0)
    assert torch.isnan(one).all()


@pytest.mark.parametrize("M", [1, 8, 64, 700])
@pytest.mark.parametrize("form", ["fma", 1, 64, 128])
def test_gemm_f32_second_operand_written_by_the_kernel_in_front(M, form):
    """A product may have for its second operand what the launch before it writes: the same bits as with a wait between the two.
    Only a caller that says that no kernel writes that operand has it read early."""
    g = torch.Generator().manual_seed(M)
    N, K = 2100, 1028
    a, x = torch.randn(N, 512, generator=g).to(DEV), torch.randn(M, K, generator=g).to(DEV)
    wait, straight = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    for turn in range(4):
        b = torch.randn(K, 512, generator=g).to(DEV)
        w = torch.full((N, K), float("nan"), device=DEV)
        torch.cuda.synchronize()
        ops().gemm_f32(a, b, w, form=form)           # some hundred microseconds
        ops().gemm_f32(x, w, straight, form=form)
        torch.cuda.synchronize()
        ops().gemm_f32(x, w, wait, form=form)
        assert torch.equal(straight, wait)
        ops().gemm_f32(x, w, straight, static_weight=True, form=form)       # (written long ago by now)
        assert torch.equal(straight, wait)


def step_f32(q, k_pool, v_pool, table, pasts, counts, heads, kv_heads, hd, window, sinks=None, scratch=True, fresh=False):
    """One step as parts/attention.py runs it (``scratch=False``: without scratch, so that no sequence's keys are cut)."""
    o = ops()
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32)).to(DEV)
    keys = max(counts) if fresh else 0
    floats = o.attention_f32_scratch_floats(len(counts), heads, hd, table.shape[1], kv_heads, q.shape[0], max(counts), keys)
    out = torch.full((q.shape[0], heads * hd), float("nan"), device=DEV)
    buf = torch.full((floats + 64,), float("nan"), device=DEV) if scratch else None
    o.attention_f32(q, k_pool, v_pool, out, d(np.concatenate([[0], np.cumsum(counts)])), d(pasts), d(counts), table, max(counts), heads, kv_heads, hd,
                    window, 1.0 / math.sqrt(hd), buf, sinks=sinks, max_keys=keys)
    assert buf is None or torch.isnan(buf[floats:]).all()
    return out, floats


# Portions on a past: up to 16 rows a group (heads of the group x tokens; 2, 4, 8 and 16 rows), then tiles of 64 rows, cut along
# the keys and not; windows and chunks of positions that begin inside a page and leave some rows of a portion without a key of it.
@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 2, 128), (5, 1, 64), (8, 8, 64), (16, 1, 128), (3, 3, 128), (12, 2, 64)])
@pytest.mark.parametrize("window,sink", [(0, False), (0, True), (50, False), (200, True), (-96, False), (3, False)])
def test_attention_f32_portions(heads, kv_heads, hd, window, sink):
    pasts, most = [0, 70, 640, 129, 1000, 63, 126, 253], 40
    gen = torch.Generator().manual_seed(heads + hd + window)
    k_pool, v_pool, table, ks, vs = make_cache([p + most for p in pasts], kv_heads, hd, torch.float32, gen)
    k_pool, v_pool, table = k_pool.to(DEV), v_pool.to(DEV), table.to(DEV)
    dense_q = torch.randn(len(pasts), most, heads, hd, generator=gen)
    sinks = torch.randn(heads, generator=gen).to(DEV) if sink else None
    alone = torch.stack([step_f32(dense_q[:, t].contiguous().to(DEV), k_pool, v_pool, table, [p + t for p in pasts], [1] * len(pasts),
                                  heads, kv_heads, hd, window, sinks)[0] for t in range(most)], 1)      # single tokens
    for i, p in enumerate(pasts):
        for t in (0, 1, 2, 39):
            pos = p + t
            lo = max(0, pos - window + 1) if window > 0 else (pos // -window * -window if window < 0 else 0)
            kk, vv = (a[i][lo:pos + 1].double().repeat_interleave(heads // kv_heads, 1) for a in (ks, vs))
            s = torch.einsum("hd,jhd->hj", dense_q[i, t].double(), kk) / math.sqrt(hd)
            s = torch.cat([s, sinks.cpu().double()[:, None]], 1) if sink else s
            want = torch.einsum("hj,jhd->hd", torch.softmax(s, 1)[:, :kk.shape[0]], vv)
            torch.testing.assert_close(alone[i, t].cpu().double().view(heads, hd), want, rtol=1e-5, atol=5e-6)
    cut = 0
    for counts in ([2] * 8, [3] * 8, [1, 4, 2, 3, 1, 4, 2, 1], [8, 1, 5, 7, 8, 2, 3, 6], [16] * 8, [9, 16, 1, 12, 3, 15, 2, 5], [17, 1, 40, 33, 20, 2, 3, 31]):
        for some in (list(range(8)), [4], [2, 4]):
            own = [counts[i] for i in some]
            q = torch.cat([dense_q[i, :counts[i]] for i in some]).contiguous().to(DEV)
            want = torch.cat([alone[i, :counts[i]] for i in some])
            args = (q, k_pool, v_pool, table[some].contiguous(), [pasts[i] for i in some], own, heads, kv_heads, hd, window, sinks)
            got, floats = step_f32(*args)
            cut += floats > 0
            assert torch.equal(got, want)
            assert max(own) == 1 or torch.equal(step_f32(*args, scratch=False)[0], want)
    assert cut
    got = step_f32(dense_q[0].contiguous().to(DEV), k_pool, v_pool, table[:1].contiguous(), [0], [most], heads, kv_heads, hd, window, sinks, fresh=True)[0]
    assert torch.equal(got, alone[0])


def test_attention_f32_many_sequences_need_no_scratch():
    """A batch that fills the GPU with a block a (sequence, kv head): the same bits as each sequence by itself."""
    heads, kv_heads, hd, n = 16, 8, 64, 80
    gen = torch.Generator().manual_seed(5)
    pasts = [(37 * i) % 500 for i in range(n)]
    k_pool, v_pool, table, _, _ = make_cache([p + 1 for p in pasts], kv_heads, hd, torch.float32, gen)
    k_pool, v_pool, table, q = k_pool.to(DEV), v_pool.to(DEV), table.to(DEV), torch.randn(n, heads, hd, generator=gen).to(DEV)
    got, floats = step_f32(q, k_pool, v_pool, table, pasts, [1] * n, heads, kv_heads, hd, 0)
    assert floats == 0
    for i in range(0, n, 7):
        one, floats = step_f32(q[i:i + 1].contiguous(), k_pool, v_pool, table[i:i + 1].contiguous(), pasts[i:i + 1], [1], heads, kv_heads, hd, 0)
        assert floats > 0 and torch.equal(one[0], got[i])
