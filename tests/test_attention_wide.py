"""Attention over portions with wide values (csrc/attention_wide.cu) at the edges of its tiles: 64 keys, 128 tokens, pages smaller and
larger than a key tile, windows, caps on both sides of the polynomial, garbage behind the last key."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pages(lens, past, heads, page, width, generator):
    """Shuffled pages for sequences of these lengths behind ``past`` tokens; what lies behind a sequence's last key is no number."""
    per = max(-(-(n + past) // page) for n in lens)
    pool = torch.randn(len(lens) * per, heads, page, width, generator=generator).to(torch.bfloat16)
    table = torch.randperm(len(lens) * per, generator=generator).view(len(lens), per)
    for s, n in enumerate(lens):
        for pos in range(n + past, per * page):
            pool[table[s, pos // page], :, pos % page] = float("nan")
    return pool.cuda(), table.int().cuda()


def _seen(n, past, window):
    i, j = torch.arange(past, past + n, device="cuda")[:, None], torch.arange(past + n, device="cuda")[None]
    return (j <= i) & ((i - j < window) if window else (j >= 0))


@pytest.mark.parametrize("lens,past,page,window", [([1], 0, 16, 0), ([63], 0, 8, 0), ([64], 0, 16, 0), ([65], 0, 32, 0), ([128], 64, 64, 0),
                                                   ([129], 0, 128, 0), ([300, 17, 64], 130, 16, 0), ([400], 200, 16, 100), ([257, 5], 300, 64, 64)])
@pytest.mark.parametrize("cap,sharp", [(0.0, 1.0), (0.0, 30.0), (30.0, 1.0), (15.0, 40.0)])
def test_differential_portions(lens, past, page, window, cap, sharp):
    """Against float64.  The weights are kept to 2^-17 and the sums are float, so the result is off by its own rounding to bfloat16
    (2^-8 of the value) and 2^-10 of the row's norm at most: the difference of two maps cancels some of their digits."""
    from edgerag_b200.ops import kernels

    H, G, d, dv, lam, eps, scale = 4, 2, 64, 128, 0.37, 1e-5, 0.4
    g = torch.Generator().manual_seed(sum(lens) + past)
    n = sum(lens)
    k_pages, table = _pages(lens, past, G, page, 2 * d, g)
    v_pages = torch.randn(k_pages.shape[0], G, page, dv, generator=g).to(torch.bfloat16).cuda()
    v_pages[torch.isnan(k_pages[..., :1]).expand_as(v_pages)] = float("nan")
    q = (sharp * torch.randn(n, H * 2 * d, generator=g)).to(torch.bfloat16).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(past, past + length) for length in lens]).int().cuda()
    status, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((n, H * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
    blocks = sum(-(-length // kernels.DIFF_WIDE_ROWS) for length in lens)
    kernels.diff_attention_wide(q, k_pages, v_pages, table, starts, positions, out, H, d ** -0.5, lam, eps, scale, blocks, status, window=window,
                                softcap=cap)
    assert status.item() == 0
    at = 0
    for s, length in enumerate(lens):
        rows = slice(at, at + length)
        at += length
        keys = k_pages[table[s].long()].transpose(1, 2).reshape(-1, G, 2, d)[: past + length].double()
        values = v_pages[table[s].long()].transpose(1, 2).reshape(-1, G, dv)[: past + length].double()
        for h in range(H):
            maps = []
            for m in (0, 1):
                score = q[rows].view(length, H, 2, d)[:, h, m].double() @ keys[:, h // (H // G), m].T * d ** -0.5
                score = cap * torch.tanh(score / cap) if cap else score
                maps.append(torch.softmax(score.masked_fill(~_seen(length, past, window), float("-inf")), -1) @ values[:, h // (H // G)])
            z = maps[0] - lam * maps[1]
            want = z / torch.sqrt((z * z).mean(-1, keepdim=True) + eps) * scale
            got = out[rows, h * dv: (h + 1) * dv].double()
            assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -10 * scale).all(), (s, h)
