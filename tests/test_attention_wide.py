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


@pytest.mark.parametrize("dim,rot,v,rank", [(64, 32, 64, 64), (128, 64, 128, 96), (64, 8, 128, 32), (128, 24, 64, 40)])
@pytest.mark.parametrize("lens,past,page,window", [([2], 0, 16, 0), ([64], 0, 8, 0), ([129, 2], 63, 16, 0), ([257, 128, 300], 65, 32, 0),
                                                   ([300], 200, 16, 50), ([2, 260], 400, 24, 64), ([256], 1, 16, 100)])
def test_latent_portions_over_rows(dim, rot, v, rank, lens, past, page, window):
    """Gather, turned queries and the attention over up-projected rows, from the second row of a batch on, with sinks and gates, against float64
    on the rows that the product left: weights to 2^-17 and float sums, rounded once to bfloat16 (2^-8 of the value; 2^-13 of the
    values' size where they cancel)."""
    from edgerag_b200.ops import kernels

    H, scale, first = 3, 0.11, 1
    g = torch.Generator().manual_seed(sum(lens) + dim)
    rand = lambda *shape: torch.randn(*shape, generator=g)      # noqa: E731
    pages, table = _pages(lens, past, 1, page, rank + rot, g)
    n = first + sum(lens)
    for s, length in enumerate(lens):                           # pages that a window has left behind hold no numbers either
        for pos in range(0, max(0, past - window + 1) // page * page if window else 0):
            pages[table[s, pos // page].long(), :, pos % page] = float("nan")
    starts = torch.tensor([first, *(first + torch.tensor(lens).cumsum(0)).tolist()], dtype=torch.int32).cuda()
    positions = torch.cat([torch.zeros(first, dtype=torch.long)] + [torch.arange(past, past + length) for length in lens]).int().cuda()
    q = (2.0 * rand(n, H * (dim + rot) + 8)).to(torch.bfloat16).cuda()[:, : H * (dim + rot)]
    gate, sink = rand(n, H).to(torch.bfloat16).cuda(), (3.0 * rand(H)).cuda()
    inv_freq = (10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64) * 2 / rot)).float().cuda()
    rows = past + max(lens) if not window else min(past + max(lens), window + max(lens) + 63)
    rows = -(-rows // 64) * 64
    latents = torch.empty(len(lens) * rows, rank + rot, dtype=torch.bfloat16, device="cuda")
    kernels.latent_gather(pages, table, starts, positions, latents, rows, window)
    q_rot = torch.empty(n, H, 64, dtype=torch.bfloat16, device="cuda")
    kernels.latent_q_rows(q, positions, inv_freq, H, dim, rot, rot, q_rot, rot_mult=1.1)
    kv = torch.empty(len(lens) * rows, H * (dim + v), dtype=torch.bfloat16, device="cuda")
    kernels.linear(latents[:, :rank], (rand(H * (dim + v), rank) / rank ** 0.5).to(torch.bfloat16).cuda(), kv)
    out, status = torch.full((n, H, v), float("nan"), dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    kernels.latent_attention_wide(q, q_rot, kv, latents, starts, positions, out, dim, rot, scale, rows,
                                  sum(-(-length // kernels.LATENT_WIDE_ROWS) for length in lens), status, gate=gate, sink=sink, window=window)
    assert status.item() == 0 and torch.isnan(out[:first]).all()
    angle = positions.double()[:, None] * inv_freq.double()
    turned = q.reshape(n, H, dim + rot)[..., dim:].double()
    pairs = torch.stack([turned[..., 0::2] * angle.cos()[:, None] - turned[..., 1::2] * angle.sin()[:, None],
                         turned[..., 1::2] * angle.cos()[:, None] + turned[..., 0::2] * angle.sin()[:, None]], -1).flatten(-2) * 1.1
    assert (q_rot[..., :rot].double() - pairs).abs().max() < 2.0 ** -8 * pairs.abs().max() and not q_rot[..., rot:].any()
    at = first
    for s, length in enumerate(lens):
        lo = max(0, past - window + 1) if window else 0
        base, n_keys, t = lo // 64 * 64, past + length - lo, slice(at, at + length)
        keys = slice(s * rows + lo - base, s * rows + lo - base + n_keys)
        flat = pages[table[s].long()].reshape(-1, rank + rot)[lo: past + length]
        assert torch.equal(latents[keys], flat) and not latents[s * rows: keys.start].any() and not latents[keys.stop: (s + 1) * rows].any()
        seen = _seen(length, past, window)[:, lo:]
        for h in range(H):
            k = torch.cat([kv[keys, h * (dim + v): h * (dim + v) + dim], latents[keys, rank:]], 1).double()
            value = kv[keys, h * (dim + v) + dim: (h + 1) * (dim + v)].double()
            query = torch.cat([q.reshape(n, H, dim + rot)[t, h, :dim], q_rot[t, h, :rot]], 1).double()
            score = (query @ k.T * scale).masked_fill(~seen, float("-inf"))
            weight = torch.softmax(torch.cat([score, sink[h].double().expand(length, 1)], 1), -1)[:, :-1]
            want = weight @ value * torch.sigmoid(gate[t, h].double())[:, None]
            assert ((out[t, h].double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -13 * value.abs().max()).all(), (s, h)
        at += length


@pytest.mark.parametrize("lens", [[127], [128], [3, 1, 2, 130], [1] * 129])
@pytest.mark.parametrize("rot_dims", [0, 32])
def test_differential_rows_by_eight_channels(lens, rot_dims):
    """The convolution, rotation and cache write around the line between the kernels (128 tokens), against float64: float sums of four
    terms, turned in float, rounded once to bfloat16 (2^-8 of the value; angles of up to 200 in float: 2^-16 of the channel's size)."""
    from edgerag_b200.ops import kernels

    H, G, d, dv, page, n = 2, 1, 32, 24, 16, sum(lens)
    channels = (H + G) * 2 * d + G * dv
    g = torch.Generator().manual_seed(n + rot_dims)
    rand = lambda *shape: torch.randn(*shape, generator=g)      # noqa: E731
    proj, weight, record = rand(n, channels + 4).to(torch.bfloat16).cuda(), (0.4 * rand(channels, 4)).cuda(), rand(len(lens) + 1, 3, channels).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    seq = torch.tensor([s for s, length in enumerate(lens) for _ in range(length)], dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(70, 70 + length) for length in lens]).int().cuda()
    held, slots = torch.arange(len(lens), 0, -1, dtype=torch.int32).cuda(), torch.randperm(n + 8, generator=g)[:n].int()
    slots[n // 2] = -1
    k_pages = torch.zeros((n + 8) // page + 1, G, page, 2 * d, dtype=torch.bfloat16, device="cuda")
    v_pages = torch.zeros(k_pages.shape[0], G, page, dv, dtype=torch.bfloat16, device="cuda")
    q = torch.empty(n, H * 2 * d, dtype=torch.bfloat16, device="cuda")
    freq = (1000.0 ** (-torch.arange(d // 2) / (d // 2))).float().cuda()
    kernels.diff_prepare(proj, q, positions, H, G, d, dv, inv_freq=freq if rot_dims else None, rot_dims=rot_dims, conv_w=weight, conv_state=record,
                         seq_of_token=seq, seq_starts=starts, state_slots=held, slots=slots.cuda(), k_pages=k_pages, v_pages=v_pages, page_size=page)
    want = torch.cat([sum(torch.cat([record[held[s]].double(), proj[starts[s]: starts[s + 1], :channels].double()], 0)[j: j + length] * weight[:, j].double()
                          for j in range(4)) for s, length in enumerate(lens)], 0)
    maps = want[:, : (H + G) * 2 * d].reshape(n, -1, d)
    if rot_dims:
        a = (positions.double()[:, None] * freq.double())[:, None]
        lo, hi = maps[..., : d // 2], maps[..., d // 2:]
        maps = torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)
    close = lambda got, exact: ((got.double() - exact).abs() <= exact.abs() * 2.0 ** -8 + 2.0 ** -14).all()      # noqa: E731
    maps = maps.reshape(n, -1)
    assert close(q, maps[:, : H * 2 * d])
    kept = slots >= 0
    at = slots[kept].long().cuda()
    assert close(k_pages[at // page, 0, at % page], maps[kept.cuda(), H * 2 * d:]) and close(v_pages[at // page, 0, at % page], want[kept.cuda(), -dv:])
    assert int((k_pages.abs().sum(-1) > 0).sum()) == int(kept.sum())


@pytest.mark.parametrize("lens", [[128], [3, 1, 2, 250]])
@pytest.mark.parametrize("rot_dims", [0, 64])
def test_differential_rows_have_the_bits_of_the_general_kernel(lens, rot_dims):
    """Rows whose length is no multiple of four take the general kernel: the same numbers in such rows give the same bits."""
    from edgerag_b200.ops import kernels

    H, G, d, dv, page, n = 4, 2, 64, 128, 16, sum(lens)
    channels = (H + G) * 2 * d + G * dv
    g = torch.Generator().manual_seed(n + rot_dims)
    rand = lambda *shape: torch.randn(*shape, generator=g)      # noqa: E731
    proj, weight, record = rand(n, channels + 6).to(torch.bfloat16).cuda(), (0.4 * rand(channels, 4)).cuda(), rand(len(lens), 3, channels).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    seq = torch.tensor([s for s, length in enumerate(lens) for _ in range(length)], dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(70, 70 + length) for length in lens]).int().cuda()
    freq = (1000.0 ** (-torch.arange(d // 2) / (d // 2))).float().cuda()
    results = []
    for rows in (proj[:, :channels].contiguous(), proj):
        k_pages = torch.zeros(n // page + 1, G, page, 2 * d, dtype=torch.bfloat16, device="cuda")
        v_pages = torch.zeros(n // page + 1, G, page, dv, dtype=torch.bfloat16, device="cuda")
        q = torch.empty(n, H * 2 * d, dtype=torch.bfloat16, device="cuda")
        kernels.diff_prepare(rows, q, positions, H, G, d, dv, inv_freq=freq if rot_dims else None, rot_dims=rot_dims, conv_w=weight, conv_state=record,
                             seq_of_token=seq, seq_starts=starts, state_slots=torch.arange(len(lens), dtype=torch.int32).cuda(),
                             slots=torch.arange(n, dtype=torch.int32).cuda(), k_pages=k_pages, v_pages=v_pages, page_size=page)
        results.append((q, k_pages, v_pages))
    assert all(torch.equal(a, b) for a, b in zip(*results))
