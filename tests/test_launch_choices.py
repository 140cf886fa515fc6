"""Host-side choices that the kernels' launches rest on, checked without a GPU: how many slices the single-token
attention cuts a sequence into, and when a product normalises its own input."""

import ctypes

import pytest
import torch

from sleuth_b200.kernels import ops
from sleuth_b200.parts import linear

SMS = 148


@pytest.mark.parametrize("kv_heads,group", [(8, 2), (2, 4), (1, 16), (4, 40), (16, 1)])
@pytest.mark.parametrize("table_stride", [1, 4, 8, 64, 512])
def test_decode_slices_fill_one_round_and_never_more(kv_heads, group, table_stride):
    row_tiles = (group + 15) // 16
    for n in list(range(1, 70)) + [100, 300]:
        blocks = n * kv_heads * row_tiles
        s = ops.decode_splits(n, kv_heads, group, table_stride, sms=148)
        assert s >= 1
        # a slice holds at least four pages of the longest sequence, unless one slice per pair is all there is
        assert s == 1 or s <= max(1, table_stride // 4) or s == 2
        if blocks <= 2 * SMS:
            # everything runs at once: with three page buffers two blocks fit an SM, with two buffers three
            assert s * blocks <= 3 * SMS
        else:
            assert s == 1 or s * blocks <= 3 * SMS
        # it depends on the batch and the table's width only: the same answer again
        assert s == ops.decode_splits(n, kv_heads, group, table_stride, sms=148)


def test_decode_slices_at_the_benchmark_shapes():
    # 8 kv heads, 2 query heads each, sequences of up to 4,096 keys (64 pages)
    assert ops.decode_splits(1, 8, 2, 64, sms=148) == 16      # capped: four pages a slice
    assert ops.decode_splits(8, 8, 2, 64, sms=148) == 6       # 384 blocks with two page buffers, not 256 with three
    assert ops.decode_splits(12, 8, 2, 64, sms=148) == 3      # 4 for 3 would not pay
    assert ops.decode_splits(16, 8, 2, 64, sms=148) == 3
    assert ops.decode_splits(64, 8, 2, 64, sms=148) == 1


def test_norm_is_fused_only_where_it_was_measured_to_pay():
    assert linear.use_skinny(8, 4096, 1024, norm=True)
    assert linear.use_skinny(1, 4096, 2048, norm=True)
    assert not linear.use_skinny(1, 6144, 4096, norm=True)       # too wide: the norm kernel in front is faster
    assert not linear.use_skinny(16, 4096, 2048, norm=True)      # too many rows for that width
    assert linear.use_skinny(16, 6144, 4096)                     # the plain product still takes it
    assert not linear.use_skinny(linear.SKINNY_ROWS + 1, 1024, 1024)


def test_timeline_groups_block_records_into_launches():
    """Two launches of one kind (the second reuses block numbers), one of another kind in between, out of order."""
    from sleuth_b200.kernels import timeline
    rec = lambda kind, block, enter, go, m2, leave: {"kind": kind, "block": block, "sm": block, "enter": enter,
                                                      "marks": [go, m2, 0], "leave": leave}
    records = [rec("gemm_skinny", 0, 100, 900, 1500, 1700), rec("gemm_skinny", 1, 120, 910, 1600, 1800),
               rec("rmsnorm", 0, 1900, 1950, 0, 2500),
               rec("gemm_skinny", 0, 2000, 2900, 3300, 3500), rec("gemm_skinny", 1, 2600, 2950, 3400, 3600)]
    records.sort(key=lambda r: r["enter"])
    out = timeline.launches(records)
    assert [(L["kind"], L["blocks"]) for L in out] == [("gemm_skinny", 2), ("rmsnorm", 1), ("gemm_skinny", 2)]
    first, norm, second = out
    assert (first["first_enter"], first["last_enter"], first["first_go"], first["last_go"]) == (100, 120, 900, 910)
    assert (first["last_mark2"], first["first_leave"], first["last_leave"]) == (1600, 1700, 1800)
    assert norm["last_mark2"] == 0 and norm["last_leave"] == 2500
    assert (second["first_enter"], second["last_enter"], second["last_leave"]) == (2000, 2600, 3600)


def test_single_token_attention_has_two_page_buffers_where_they_were_faster():
    """Where all blocks are resident with two and not with three, and at heads of 128 from the third round on."""
    stages = lambda hd, blocks: ops.lib().dll.slb_attention_decode_stages(hd, ctypes.c_longlong(blocks), SMS)
    assert [stages(128, b) for b in (8, 296, 297, 444, 445, 512, 592, 593, 640, 1024, 2048)] == [3, 3, 2, 2, 3, 3, 3, 2, 2, 2, 2]
    assert [stages(64, b) for b in (8, 296, 297, 444, 445, 512, 593, 1024, 2048)] == [3, 3, 2, 2, 3, 3, 3, 3, 3]


def test_sampler_blocks_fill_their_sm():
    """Few rows: a block an SM, as large as it can be; more rows: two blocks of half the size."""
    threads = ops.lib().dll.slb_sample_threads
    assert threads(1) == threads(18) == 1024 and threads(19) == threads(64) == 512
    lean = ops.lib().dll.slb_sample_threads_of
    assert lean(18, 151936, 50) == lean(37, 8000, 50) == 512 and lean(38, 151936, 50) == lean(64, 8000, 1) == 256
    assert lean(17, 151936, 50) == 1024 and lean(64, 151936, 51) == lean(64, 7999, 50) == 512


def test_float32_attention_scratch():
    """Scratch of the 32-bit attention: none where blocks have a sequence to themselves, never more than 256 MB, never more than the
    form that every single-token step could have needed, and the same for every replay of a step's shape."""
    f = ops.attention_f32_scratch_floats
    wide = 640                                     # 40,960 keys
    assert f(256, 16, 128, wide, 8) == f(64, 16, 64, wide, 8) == f(64, 32, 64, wide, 8, 128, 2) == 0      # blocks enough without cutting
    assert f(591, 16, 128, wide, 1) == 0           # would be 1.5 GB
    for n in (1, 2, 8, 30, 64, 100, 300):
        for heads, kv in ((16, 8), (16, 1), (32, 8), (8, 8)):
            for stride in (1, 2, 3, 64, wide):
                assert 0 <= f(n, heads, 128, stride, kv) <= min(f(n, heads, 128, stride), 1 << 26)
                for count in (1, 2, 5, 20, 64, 300):
                    assert 0 <= f(n, heads, 128, stride, kv, n * count, count) <= 1 << 26
    assert f(1, 16, 128, 64, 8) == 16 * 32 * 130
    assert f(1, 16, 128, 64, 8, 20, 20) == 20 * 16 * 32 * 130        # a second turn: 8 tiles, cut along the keys
    assert f(1, 16, 128, 64, 8, 100, 100, 100) == 0                  # a prompt of one chunk
    assert f(8, 16, 128, 64, 8, 3200, 400) == 0                      # tiles enough


def test_float32_fma_product_takes_what_was_faster():
    """Products at which the FMA kernels, the streaming one (0) and the tiles (8, 6 or 4 rows a thread), were timed on a B200, of matrices
    that do not go to the tensor cores."""
    choice = ops.lib().dll.slb_gemm_f32_choice
    for M, N, K, vec, want in [(128, 6144, 160, 1, 8), (600, 503, 160, 1, 4), (48, 32768, 160, 1, 8), (32, 32768, 96, 1, 8), (16, 32768, 96, 1, 0),
                               (600, 1024, 77, 0, 8), (128, 6144, 77, 0, 8), (64, 503, 77, 0, 0), (80, 1024, 1030, 0, 0), (1500, 503, 1030, 0, 8), (12, 32768, 1030, 0, 0)]:
        assert not ops.f32_on_tensor_cores(N, K, 0 if vec else 4)
        assert (choice(M, N, K, vec) == 0) == (want == 0), (M, N, K, choice(M, N, K, vec))
    assert choice(600, 503, 160, 1) == 4


def test_large_matrices_of_some_rows_are_streamed_through_the_tensor_cores():
    """Where products and whole runs were timed with and without (4B, 8B and 0.6B sizes, and such between them)."""
    for M, N, K, gated, want in [(16, 2560, 9728, False, True), (16, 9728, 2560, True, True), (24, 6144, 2560, False, True), (64, 12288, 4096, True, True),
                                 (8, 9728, 2560, True, False), (65, 12288, 4096, True, False), (24, 1024, 3072, False, False), (24, 3072, 1024, True, False),
                                 (16, 151936, 2560, False, False), (24, 151936, 2560, False, True), (16, 4096, 2560, False, False), (16, 4096, 4096, False, False), (16, 2560, 4096, False, True), (16, 2048, 8192, False, False),
                              (16, 6144, 2560, False, True), (16, 3072, 4096, True, False), (16, 6144, 2560, True, True), (32, 4096, 2048, False, True), (33, 6144, 2560, False, False),
                              (64, 8192, 2048, False, False), (64, 4096, 12288, False, True), (64, 9728, 2560, True, False), (48, 9728, 2560, True, True), (64, 4608, 1024, True, True)]:
        assert linear.use_stream(M, N, K, gated) == want, (M, N, K)


def test_rows_that_lie_otherwise_stay_with_the_other_kernels():
    """The streaming kernel reads rows one behind the other from 16-byte boundaries on; strided rows and odd addresses go on as before."""
    w = torch.empty(4096 * 2560 + 8, dtype=torch.bfloat16)
    weight, shifted = w[:4096 * 2560].view(4096, 2560), w[1:4096 * 2560 + 1].view(4096, 2560)
    wide = torch.empty(20, 2568, dtype=torch.bfloat16)
    h = torch.empty(20 * 2560 + 1, dtype=torch.bfloat16)
    assert linear.streams(h[:-1].view(20, 2560), weight) and linear.streams(h[:-1].view(20, 2560), weight, gated=True)
    assert not linear.streams(h[1:].view(20, 2560), weight) and not linear.streams(h[:-1].view(20, 2560), shifted)
    assert not linear.streams(wide[:, :2560], weight)


def test_float32_product_on_the_tensor_cores_takes_what_was_faster():
    """Forms at which products were timed on a B200 (1: the kernel for few rows; else tokens of a tile), and the matrices that go there."""
    form = ops.f32_form
    for M, N, K, want in [(1, 4096, 1024, 1), (8, 19456, 2560, 1), (1, 151936, 1024, 1), (16, 1024, 3072, 1), (32, 6144, 1024, 1), (64, 1024, 2048, 1), (16, 151936, 1024, 32),
                          (64, 6144, 1024, 64), (1500, 4096, 1024, 128), (1500, 1024, 3072, 128)]:
        assert form(M, N, K) == want, (M, N, K, form(M, N, K))
    assert ops.f32_on_tensor_cores(512, 1024, 0) and not ops.f32_on_tensor_cores(4096, 1020, 0) and not ops.f32_on_tensor_cores(511, 4096, 0)
    assert not ops.f32_on_tensor_cores(512, 1030, 0) and not ops.f32_on_tensor_cores(512, 1024, 8)


def test_prompts_of_padded_heads_where_they_were_faster():
    """Row widths of latent attention's whole prompts: head sizes, heads and longest sequences at which both ways were timed."""
    from types import SimpleNamespace as N
    from sleuth_b200.parts.latent_attention import LatentAttention
    part = object.__new__(LatentAttention)
    part.ctx = N(dtype=torch.bfloat16)
    for heads, dn, P, dv, longest, want in [(16, 64, 32, 64, 2048, 128), (16, 40, 16, 40, 512, 64), (32, 64, 32, 64, 128, 128), (16, 64, 32, 64, 100, 0), (128, 64, 32, 64, 128, 0),
                                            (128, 64, 32, 64, 512, 128), (16, 128, 64, 128, 2048, 0), (16, 60, 16, 64, 2048, 0), (16, 128, 0, 64, 2048, 128)]:
        part.spec = N(heads=heads, plain_dim=dn, rot_dim=P, value_dim=dv, scale=0.1)
        assert part._prompt_row_width(N(max_count=longest)) == want, (heads, dn, P, dv, longest)
