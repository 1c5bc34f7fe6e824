"""The router over many tokens at once: its choices, weights and side gate against the router over fewer tokens (the same sums in the
same order, so the same bits) and against float64, the experts' lists against a count on the host, and the experts' products in tiles of 256 rows against smaller ones."""

from __future__ import annotations

import pytest
import torch

from edgerag_b200.ops import kernels as K


def _route(x, router, top, tile, gate, **how):
    n, rows = x.shape[0], router.shape[0]
    experts = rows - int(gate)
    lists = torch.full((K.moe_lists_ints(n, experts, top),), -7, dtype=torch.int32, device="cuda")
    score = torch.full((n * top,), float("nan"), device="cuda")
    side = torch.full((n,), float("nan"), device="cuda") if gate else None
    K.moe_route(x, router, top, lists, score, tile, side_gate=side, **how)
    torch.cuda.synchronize()
    return [v.cpu() for v in K._moe_lists(lists, n, experts, top)], score.cpu(), side.cpu() if gate else None


def _check_lists(parts, experts, tile):
    choice, order, counts, offsets, tiles = (v.long() for v in parts)
    want = torch.bincount(choice, minlength=experts)
    assert torch.equal(counts[:experts], want)
    assert torch.equal(offsets, torch.cat([want.new_zeros(1), want.cumsum(0)]))
    assert torch.equal(tiles, torch.cat([want.new_zeros(1), (-(-want // tile)).cumsum(0)]))
    assert torch.equal(order, torch.argsort(choice, stable=True))


@pytest.mark.gpu
@pytest.mark.parametrize("n,experts,top,width,gate", [
    (1024, 32, 4, 2048, True), (1025, 5, 1, 128, False), (1039, 7, 3, 384, True), (1024, 130, 6, 1024, False), (2371, 33, 2, 256, True),
])
def test_many_tokens_route_as_few(n, experts, top, width, gate):
    g = torch.Generator().manual_seed(n + experts)
    wide = torch.randn(n, width + 8, generator=g).to(torch.bfloat16).cuda()
    x = wide[:, :width]                                               # (rows with a stride of their own)
    router = (torch.randn(experts + int(gate), width, generator=g) * width ** -0.5).cuda()
    parts, score, side = _route(x, router, top, 128, gate)
    _check_lists(parts, experts, 128)
    for a in range(0, n, 500):                                        # the kernel for fewer tokens
        some, some_score, some_side = _route(x[a: a + 500], router, top, 128, gate)
        m = min(500, n - a)
        assert torch.equal(parts[0][a * top: (a + m) * top], some[0])
        assert torch.equal(score[a * top: (a + m) * top], some_score)
        assert not gate or torch.equal(side[a: a + m], some_side)
    z = x.cpu().double() @ router.cpu().double().T
    # |error of a float sum of `width` products| <= width * 2^-24 * sum |x w|; a sigmoid's slope is at most 1/4, plus its own rounding
    bound = width * 2.0 ** -24 * (x.cpu().double().abs() @ router.cpu().double().abs().T).max() / 4 + 2.0 ** -21
    got = torch.gather(torch.sigmoid(z), 1, parts[0].long().view(n, top))
    assert (got.view(-1) - score.double()).abs().max() <= bound
    assert not gate or (torch.sigmoid(z[:, experts]) - side.double()).abs().max() <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("n,experts,top", [(1, 1, 1), (3, 2, 2), (127, 4, 1), (129, 300, 3), (500, 513, 2), (513, 700, 1), (2049, 9, 4)])
def test_lists_of_any_size(n, experts, top):
    g = torch.Generator().manual_seed(n)
    x = torch.randn(n, 64, generator=g).to(torch.bfloat16).cuda()
    router = torch.randn(experts, 64, generator=g).cuda()
    router[0] = 0.0                                                   # (and every weight alike for some rows: one long list)
    x[: n // 2] = 0.0
    for tile in (16, 128):
        parts, _, _ = _route(x, router, top, tile, False)
        _check_lists(parts, experts, tile)


@pytest.mark.gpu
@pytest.mark.parametrize("counts,width,ff", [
    ((1, 16, 17, 64, 65, 128, 129, 0), 64, 128), ((255, 256, 257, 511), 136, 72), ((300, 0, 520), 512, 264), ((240,), 72, 8),
])
def test_products_in_tiles_of_256_rows(counts, width, ff):
    """A row's product does not depend on the tile that it falls into: the same bits in tiles of 256 rows as in tiles of 32; and close to float64."""
    g = torch.Generator().manual_seed(sum(counts))
    n, experts = sum(counts), len(counts)
    which = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(n, generator=g)]
    x = torch.zeros(n, 64)
    x[torch.arange(n), which] = 1.0
    xs = torch.randn(n, width, generator=g).to(torch.bfloat16).cuda()
    w_in = (torch.randn(experts, 2 * ff, width, generator=g) * width ** -0.5).to(torch.bfloat16).cuda()
    w_out = (torch.randn(experts, width, ff, generator=g) * ff ** -0.5).to(torch.bfloat16).cuda()
    single = w_in[:, :ff].contiguous()
    got = {}
    for tile in (32, 256):
        lists = torch.zeros(K.moe_lists_ints(n, experts, 1), dtype=torch.int32, device="cuda")
        score = torch.empty(n, device="cuda")
        K.moe_route(x.to(torch.bfloat16).cuda(), 20.0 * torch.eye(experts, 64, device="cuda"), 1, lists, score, tile)
        act, act1 = (torch.full((n, ff), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        parts = torch.full((1, n, width), float("nan"), device="cuda")
        K.moe_tc_gate_up(xs, w_in, lists, 1, tile, act)
        K.moe_tc_up_act(xs, single, lists, 1, tile, act1)
        K.moe_tc_down(act, w_out, lists, 1, tile, parts)
        got[tile] = (act.cpu(), act1.cpu(), parts.cpu())
        order = K._moe_lists(lists, n, experts, 1)[1].long().cpu()
    assert all(torch.equal(a, b) for a, b in zip(got[32], got[256]))
    act, _, parts = (v.double() for v in got[256])
    rows = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))          # (the lists' rows stand in the experts' order)
    w = w_out.cpu().double()[rows]
    want = torch.einsum("nf,nhf->nh", act, w)
    # float sums of ff products: their error is at most ff * 2^-24 * sum |act w| (the unit may cut instead of rounding: twice that)
    bound = 2 * ff * 2.0 ** -24 * torch.einsum("nf,nhf->nh", act.abs(), w.abs()).max() + 1e-30
    assert (parts[0][order] - want).abs().max() <= bound
