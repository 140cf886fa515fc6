"""The routed experts of a step of few pairs on the tensor cores (csrc/moe.cu, moe_few_*_mma_kernel) against float64: experts
that many tokens share (more than the sixteen rows of an instruction), the most pairs there are, columns that fill no group of 8,
widths whose parts for the warps are uneven or empty, identity experts, further rows, an empty target."""

import pytest
import torch

from sleuth_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tokens,top,E,dim,ff", [(1, 1, 3, 32, 32), (1, 6, 64, 2048, 1408), (3, 2, 4, 96, 352), (32, 2, 3, 256, 64), (64, 1, 2, 160, 96),
                                                 (16, 4, 5, 1024, 768), (8, 8, 40, 544, 32), (21, 3, 7, 64, 1056)])
@pytest.mark.parametrize("identity,store,further", [(0, False, False), (2, False, True), (1, True, False)])
def test_few_pairs(tokens, top, E, dim, ff, identity, store, further):
    if top > E + identity:
        pytest.skip("more choices than experts")
    g = torch.Generator().manual_seed(tokens * 100 + dim + identity)
    h = torch.randn(tokens, dim, generator=g).bfloat16()
    w_gu, w_down = torch.randn(E, 2 * ff, dim, generator=g).div(dim ** 0.5).bfloat16(), torch.randn(E, dim, ff, generator=g).div(ff ** 0.5).bfloat16()
    choice = torch.stack([torch.randperm(E + identity, generator=g)[:top] for _ in range(tokens)]).int()
    weight, x0, more = torch.rand(tokens, top, generator=g), torch.randn(tokens, dim, generator=g), torch.randn(tokens, dim, generator=g)
    want, size = torch.zeros(tokens, dim, dtype=torch.float64), torch.zeros(tokens, dim, dtype=torch.float64)
    for t in range(tokens):
        for k in range(top):
            e, row = int(choice[t, k]), h[t].double()
            if e < E:
                up = w_gu[e].double() @ row
                act = (torch.nn.functional.silu(up[:ff]) * up[ff:]).bfloat16().double()      # held in the run's dtype
                row = w_down[e].double() @ act
                size[t] += weight[t, k].double() * (w_down[e].double().abs() @ act.abs())
            want[t] += weight[t, k].double() * row
    want += (0 if store else x0.double()) + (more.double() if further else 0)
    d = lambda a: a.to(DEV).contiguous()
    x = d(x0)
    pairs = tokens * top
    act, y = torch.empty(pairs, ff, device=DEV, dtype=torch.bfloat16), torch.empty(pairs, dim, device=DEV)
    ints = torch.zeros(max(pairs, E + identity), dtype=torch.int32, device=DEV)
    ops.moe_experts(d(h), d(w_gu), d(w_down), ints[:E + identity], ints[:pairs], d(weight.view(-1)), act, y, x, top, "silu", None, d(choice.view(-1)),
                    ints[:pairs], extra=d(more) if further else None, identity=identity, store=store)
    # 32-bit sums differ in their order; now and then an activation rounds to the neighbouring bfloat16 (2^-8 of its size)
    got = x.cpu().double()
    assert ((got - want).abs() <= 2.0 ** -8 * size + 1e-5 * (1 + want.abs())).all()
    assert float((got - want).norm() / want.norm()) < 1e-3


# The same where the tensor-core kernels run (matrices of 512 x 512 values and more): two, four and eight parts of the width with an
# uneven last one, one, two and four parts of the experts' width, column groups that are not full, more than 16 and 32 rows an expert.
@pytest.mark.parametrize("tokens,top,E,dim,ff", [(32, 2, 3, 544, 512), (64, 1, 2, 512, 544), (21, 3, 7, 1056, 288), (5, 2, 6, 2080, 160), (8, 8, 40, 512, 1056),
                                                 (4, 3, 5, 160, 2080), (16, 4, 20, 1024, 2112), (1, 8, 64, 4096, 512), (40, 1, 1, 992, 1088)])
@pytest.mark.parametrize("identity,store,further", [(0, False, False), (2, False, True), (1, True, False)])
def test_few_pairs_on_the_tensor_cores(tokens, top, E, dim, ff, identity, store, further):
    test_few_pairs(tokens, top, E, dim, ff, identity, store, further)


@pytest.mark.parametrize("top,E,dim,ff", [(6, 64, 2048, 1408), (4, 16, 1024, 768), (2, 8, 512, 3584), (2, 4, 256, 128)])
def test_a_tokens_bits_do_not_depend_on_the_tokens_beside_it(top, E, dim, ff):
    g = torch.Generator().manual_seed(dim + ff)
    n = 64 // top
    d = lambda a: a.to(DEV).contiguous()
    h = d(torch.randn(n, dim, generator=g).bfloat16())
    w_gu, w_down = d(torch.randn(E, 2 * ff, dim, generator=g).div(dim ** 0.5).bfloat16()), d(torch.randn(E, dim, ff, generator=g).div(ff ** 0.5).bfloat16())
    choice, weight = d(torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(n)]).int()), d(torch.rand(n, top, generator=g))

    def run(a, b):
        x, pairs = torch.zeros(b - a, dim, device=DEV), (b - a) * top
        act, y = torch.empty(pairs, ff, device=DEV, dtype=torch.bfloat16), torch.empty(pairs, dim, device=DEV)
        ints = torch.zeros(max(pairs, E), dtype=torch.int32, device=DEV)
        ops.moe_experts(h[a:b], w_gu, w_down, ints[:E], ints[:pairs], weight[a:b].reshape(-1), act, y, x, top, "silu", None, choice[a:b].reshape(-1), ints[:pairs])
        return x

    together = run(0, n)
    for a, b in ((0, 1), (1, 3), (n - 1, n), (n // 2, n)):
        assert torch.equal(run(a, b), together[a:b])
