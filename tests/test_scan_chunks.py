"""The recurrent mixers' kernels that take a portion 64 tokens at a time, at the sizes where they can go wrong: a token beside
a chunk's end, the smallest and largest states, single tokens beside portions, decays of almost nothing and almost one."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ssm_reference(xbc, dt_raw, dt_bias, a_log, skip, state, H, P, N, G):
    n, inner = xbc.shape[0], H * P
    x = xbc.double()
    u = x[:, :inner].view(n, H, P)
    B = x[:, inner: inner + G * N].view(n, G, N).repeat_interleave(H // G, 1)
    C = x[:, inner + G * N:].view(n, G, N).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt_raw.double() + dt_bias.double(), threshold=1e9)
    decay, S, y = torch.exp(-torch.exp(a_log.double()) * dt), state.double().clone(), torch.empty_like(u)
    for t in range(n):
        S = S * decay[t, :, None, None] + (dt[t, :, None] * B[t])[:, :, None] * u[t][:, None, :]
        y[t] = torch.bmm(C[t][:, None], S)[:, 0]
    return (y + skip.double()[:, None] * u).reshape(n, inner), S


@pytest.mark.parametrize("H,P,N,G", [(4, 32, 32, 2), (2, 64, 64, 1), (4, 64, 128, 2)])
@pytest.mark.parametrize("lens", [[63], [64], [65], [2], [1, 129, 1], [130, 3, 64, 1, 17]])
@pytest.mark.parametrize("pace", [-6.0, 0.0, 4.0])
def test_state_space_chunks(H, P, N, G, lens, pace):
    """Chunks and the walk against float64.  Both are float throughout (a product's operands go in whole, as three pieces), so
    each entry is within a few hundred roundings of 2^-24 of the largest of the row of sums it belongs to: 3e-5 of the
    largest result, the band of the tests of the walk."""
    from edgerag_b200.ops import kernels

    n, slots = sum(lens), [len(lens) - i for i in range(len(lens))]
    g = torch.Generator().manual_seed(N + n)
    inner = H * P
    xbc = (torch.randn(n, inner + 2 * G * N, generator=g) * 0.5).to(torch.bfloat16).cuda()
    proj = torch.randn(n, 8, generator=g).to(torch.bfloat16).cuda()
    dt_bias, a_log, skip = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda() * 0.3 + pace, torch.randn(H, generator=g).cuda()
    before = torch.randn(len(lens) + 1, H, N, P, generator=g).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    for longest in (1 << 20, 1):                 # portions in chunks (the largest the rule accepts), every token by the walk
        state, y = before.clone(), torch.full((n, inner), float("nan"), device="cuda")
        kernels.ssm_scan(xbc, proj, 1, dt_bias, a_log, skip, state, len(lens), starts, torch.tensor(slots, dtype=torch.int32).cuda(), y, G,
                         longest=longest)
        at = 0
        for s, length in enumerate(lens):
            rows = slice(at, at + length)
            want_y, want_s = _ssm_reference(xbc[rows], proj[rows, 1: 1 + H], dt_bias, a_log, skip, before[slots[s]], H, P, N, G)
            assert (y[rows].double() - want_y).abs().max() < 3e-5 * max(1.0, want_y.abs().max()), (s, longest)
            assert (state[slots[s]].double() - want_s).abs().max() < 3e-5 * max(1.0, want_s.abs().max()), (s, longest)
            # in chunks a few roundings in the mean: operands in two pieces instead of three would be off by some 2^-18 each, 2e-6 in the mean.
            # (The walk rounds its state once a token, n 2^-25 at worst where nothing decays, which says nothing about pieces.)
            if longest > 1 and length > 1:
                assert (y[rows].double() - want_y).norm() < 6e-7 * want_y.norm() and (state[slots[s]].double() - want_s).norm() < 6e-7 * want_s.norm(), s
            at += length
        assert torch.equal(state[0], before[0])     # the slot nobody holds


def _same_as_walked(got, walked, what):
    """Numbers that are not finite lie where the walk has them and are the same; the others are within the band of the tests above."""
    assert torch.equal(torch.isfinite(got), torch.isfinite(walked)), what
    assert torch.equal(torch.nan_to_num(got[~torch.isfinite(got)]), torch.nan_to_num(walked[~torch.isfinite(walked)])), what
    fine = torch.isfinite(walked)
    assert (got[fine].double() - walked[fine].double()).abs().max() < 6e-5 * max(1.0, walked[fine].abs().max().item()), what


@pytest.mark.parametrize("P,N", [(32, 32), (64, 64), (64, 128)])
@pytest.mark.parametrize("what", ["x", "x nan", "B", "C", "step", "state", "decay"])
def test_state_space_chunks_keep_numbers_that_are_not_finite_to_the_later_tokens(P, N, what):
    """One number that is not finite at token 37 of a portion of 130 (or in its state, or a decay of exactly zero): the tokens before it
    are what they are without it, and everything is what the walk gives."""
    from edgerag_b200.ops import kernels

    H, G, lens, at = 4, 2, [1, 130, 64], 1 + 37
    n, inner, m = sum(lens), H * P, len(lens)
    g = torch.Generator().manual_seed(N)
    xbc = torch.randn(n, inner + 2 * G * N, generator=g) * 0.5
    proj, a_log = torch.randn(n, 8, generator=g), torch.randn(H, generator=g) * 0.3
    before = torch.randn(m + 1, H, N, P, generator=g)
    if what[0] in "xBC":
        xbc[at, {"x": P + 3, "B": inner + 5, "C": inner + G * N + N + 7}[what[0]]] = float("nan" if "nan" in what else "inf")
    elif what == "step":
        proj[at, 1 + 2] = float("inf")
    elif what == "state":
        before[2, 1, 9, 4] = float("inf")
    else:
        a_log[1] = 100.0
    xbc, proj = xbc.to(torch.bfloat16).cuda(), proj.to(torch.bfloat16).cuda()
    dt_bias, skip = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda()
    starts, slots = torch.tensor([0, 1, 131, 195], dtype=torch.int32).cuda(), torch.tensor([1, 2, 0], dtype=torch.int32).cuda()
    done = []
    for longest in (1 << 20, 1):
        state, y = before.clone().cuda(), torch.full((n, inner), 7.0, device="cuda")
        kernels.ssm_scan(xbc, proj, 1, dt_bias, a_log.cuda(), skip, state, m, starts, slots, y, G, longest=longest)
        done.append((y, state))
    _same_as_walked(done[0][0], done[1][0], "y")
    _same_as_walked(done[0][1], done[1][1], "state")
    y = done[0][0]
    assert torch.isfinite(y[131:]).all() and (what == "state" or torch.isfinite(y[:at]).all())
    assert torch.isfinite(y).all() == (what == "decay")


def _delta_reference(qkv, b, a, dt_bias, a_log, state, H, G, d, dv):
    n, x = qkv.shape[0], qkv.double()
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)      # noqa: E731
    q = (unit(x[:, : G * d].reshape(n, G, d)) * d ** -0.5).repeat_interleave(H // G, 1)
    k = unit(x[:, G * d: 2 * G * d].reshape(n, G, d)).repeat_interleave(H // G, 1)
    v, beta = x[:, 2 * G * d:].reshape(n, H, dv), torch.sigmoid(b.double())
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a.double() + dt_bias.double(), threshold=1e9))
    S, o = state.double().clone(), torch.empty_like(v)
    for t in range(n):
        S = S * g[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(S, k[t, :, :, None])[..., 0])
        S = S + u[:, :, None] * k[t, :, None, :]
        o[t] = torch.bmm(S, q[t, :, :, None])[..., 0]
    return o.reshape(n, H * dv), S


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 16), (4, 2, 64, 48), (2, 2, 128, 128)])
@pytest.mark.parametrize("lens", [[63], [64], [65], [2], [1, 129, 1], [130, 3, 64, 1, 17]])
@pytest.mark.parametrize("pace,alike", [(-6.0, True), (-6.0, False), (0.0, False), (4.0, False)])
def test_delta_chunks(H, G, d, dv, lens, pace, alike):
    """The delta rule in chunks and walked, against float64, with keys that resemble one another (the triangular system is
    then far from the identity) and decays of almost one and almost nothing: within the band of the walk's own test (3e-5)."""
    from edgerag_b200.ops import kernels

    n, m = sum(lens), len(lens)
    slots = [m - i for i in range(m)]
    g = torch.Generator().manual_seed(d + n)
    qkv = torch.randn(n, 2 * G * d + H * dv, generator=g) * 0.5
    if alike:
        qkv[:, G * d: 2 * G * d] = torch.randn(1, G * d, generator=g) + 0.3 * torch.randn(n, G * d, generator=g)
    qkv = qkv.to(torch.bfloat16).cuda()
    proj = torch.randn(n, 2 * H + 3, generator=g).to(torch.bfloat16).cuda()
    dt_bias, a_log = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda() * 0.3 + pace
    before = 0.3 * torch.randn(m + 1, H, dv, d, generator=g).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    for longest, room in ((1 << 20, m), (1, m), (1 << 20, 0)):      # chunks; the walk; the walk for want of scratch
        state, out = before.clone(), torch.full((n, H * dv), float("nan"), device="cuda")
        scratch = torch.full((kernels.delta_scratch_floats(n, H, G, d, dv, room),), float("nan"), device="cuda")
        kernels.delta_scan(qkv, proj, 1, 2 + H, dt_bias, a_log, state, m, starts, torch.tensor(slots, dtype=torch.int32).cuda(), out, G, d,
                           scratch, longest=longest)
        at = 0
        for s, length in enumerate(lens):
            rows = slice(at, at + length)
            want, want_s = _delta_reference(qkv[rows], proj[rows, 1: 1 + H], proj[rows, 2 + H: 2 + 2 * H], dt_bias, a_log, before[slots[s]], H, G, d, dv)
            assert (out[rows].double() - want).abs().max() < 3e-5 * max(1.0, want.abs().max()), (s, longest)
            assert (state[slots[s]].double() - want_s).abs().max() < 3e-5 * max(1.0, want_s.abs().max()), (s, longest)
            if longest > 1 and room and length > 1:      # (as for the state-space chunks; the walk's errors grow along an ill-conditioned portion)
                assert (out[rows].double() - want).norm() < 8e-7 * want.norm() and (state[slots[s]].double() - want_s).norm() < 8e-7 * want_s.norm(), s
            at += length
        assert torch.equal(state[0], before[0])


@pytest.mark.parametrize("length,walked", [(2, True), (28, True), (33, True), (300, False)])
def test_short_portions_of_the_delta_rule_are_walked(length, walked):
    """A chunk costs what 34 tokens of the walk cost: shorter portions have the walk's bits, longer ones differ from it by rounding."""
    from edgerag_b200.ops import kernels

    H, G, d, dv = 4, 4, 64, 48
    g = torch.Generator().manual_seed(length)
    qkv, proj = (torch.randn(length, w, generator=g).to(torch.bfloat16).cuda() for w in (2 * G * d + H * dv, 2 * H))
    dt_bias, a_log = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda() * 0.3
    starts, slots = torch.tensor([0, length], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()
    outs = []
    for longest in (None, 1):
        out = torch.empty(length, H * dv, device="cuda")
        kernels.delta_scan(qkv, proj, 0, H, dt_bias, a_log, torch.zeros(1, H, dv, d, device="cuda"), 1, starts, slots, out, G, d, longest=longest)
        outs.append(out)
    assert torch.equal(*outs) == walked


def test_walked_portions_do_not_depend_on_what_shares_the_step():
    """The form that ``batch_invariant`` pins (``longest`` 1): the bits of a portion alone and beside others are the same, and so is its record."""
    from edgerag_b200.ops import kernels

    g = torch.Generator().manual_seed(3)
    H, P, N, G, d, dv, lens = 4, 64, 128, 2, 128, 64, [30] + [8] * 31
    n = sum(lens)
    xbc, qkv = ((0.5 * torch.randn(n, w, generator=g)).to(torch.bfloat16).cuda() for w in (H * P + 2 * G * N, 2 * G * d + H * dv))
    proj, vec = torch.randn(n, 2 * H, generator=g).to(torch.bfloat16).cuda(), torch.randn(3, H, generator=g).cuda()
    ssm, delta = torch.randn(32, H, N, P, generator=g).cuda(), 0.3 * torch.randn(32, H, dv, d, generator=g).cuda()
    results = []
    for m in (1, 32):
        rows, starts = sum(lens[:m]), torch.tensor([0, *torch.tensor(lens[:m]).cumsum(0).tolist()], dtype=torch.int32).cuda()
        slots, states = torch.arange(m, dtype=torch.int32).cuda(), (ssm.clone(), delta.clone())
        y, o = torch.empty(rows, H * P, device="cuda"), torch.empty(rows, H * dv, device="cuda")
        kernels.ssm_scan(xbc[:rows], proj[:rows], 0, vec[0], vec[1], vec[2], states[0], m, starts, slots, y, G, longest=1)
        kernels.delta_scan(qkv[:rows], proj[:rows], 0, H, vec[0], vec[1], states[1], m, starts, slots, o, G, d, longest=1)
        results.append((y[:30], o[:30], states[0][0], states[1][0]))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("d,dv", [(64, 16), (128, 128)])
@pytest.mark.parametrize("what", ["q", "k", "v", "v nan", "strength", "decay", "state"])
def test_delta_chunks_keep_numbers_that_are_not_finite_to_the_later_tokens(d, dv, what):
    """As for the state-space chunks; a decay input of infinity is a decay of exactly zero."""
    from edgerag_b200.ops import kernels

    H, G, lens, at = 4, 2, [1, 130, 64], 1 + 37
    n, m = sum(lens), len(lens)
    g = torch.Generator().manual_seed(d + dv)
    qkv, proj = torch.randn(n, 2 * G * d + H * dv, generator=g) * 0.5, torch.randn(n, 2 * H + 3, generator=g)
    before = 0.3 * torch.randn(m + 1, H, dv, d, generator=g)
    if what[0] in "qkv":
        qkv[at, {"q": 5, "k": G * d + d + 6, "v": 2 * G * d + 3 * dv + 2}[what[0]]] = float("nan" if "nan" in what else "inf")
    elif what == "strength":
        proj[at, 1 + 2] = float("nan")
    elif what == "decay":
        proj[at, 2 + H + 1] = float("inf")
    else:
        before[2, 1, 9, 4] = float("inf")
    qkv, proj = qkv.to(torch.bfloat16).cuda(), proj.to(torch.bfloat16).cuda()
    dt_bias, a_log = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda() * 0.3
    starts, slots = torch.tensor([0, 1, 131, 195], dtype=torch.int32).cuda(), torch.tensor([1, 2, 0], dtype=torch.int32).cuda()
    done = []
    for longest in (1 << 20, 1):
        state, out = before.clone().cuda(), torch.full((n, H * dv), 7.0, device="cuda")
        kernels.delta_scan(qkv, proj, 1, 2 + H, dt_bias, a_log, state, m, starts, slots, out, G, d, longest=longest)
        done.append((out, state))
    _same_as_walked(done[0][0], done[1][0], "out")
    _same_as_walked(done[0][1], done[1][1], "state")
    out = done[0][0]
    assert torch.isfinite(out[131:]).all() and (what == "state" or torch.isfinite(out[:at]).all())
    assert torch.isfinite(out).all() == (what == "decay")


@pytest.mark.parametrize("lens", [[7], [8], [1] * 9, [255], [3, 1, 2, 250, 1], [9, 300]])
def test_short_convolution_by_eight_channels(lens):
    """Rows of four taps, with and without a bias, at counts around the lines between the kernels: float sums of five terms
    rounded once: neighbouring bfloat16 values (8 bits of significand) lie up to 2^-7 of the value apart, so rounding moves it by
    up to 2^-8 of itself, and the sums' own error is below 2^-20 of them (silu's slope is at most 1.1)."""
    from edgerag_b200.ops import kernels

    n, channels, ld, off, slots = sum(lens), 72, 96, 16, len(lens) + 1
    g = torch.Generator().manual_seed(n)
    proj = torch.randn(n, ld, generator=g).to(torch.bfloat16).cuda()
    weight, bias = torch.randn(channels, 4, generator=g).to(torch.bfloat16).cuda(), torch.randn(channels, generator=g).to(torch.bfloat16).cuda()
    record = torch.randn(slots, 3, channels, generator=g).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    seq = torch.tensor([s for s, length in enumerate(lens) for _ in range(length)], dtype=torch.int32).cuda()
    held = torch.arange(len(lens), 0, -1, dtype=torch.int32).cuda()
    for b in (bias, None):
        out = torch.full((n, channels), float("nan"), dtype=torch.bfloat16, device="cuda")
        kernels.conv_silu(proj, off, weight, b, record, seq, starts, held, out)
        at = 0
        for s, length in enumerate(lens):
            x = torch.cat([record[held[s]].double(), proj[at: at + length, off: off + channels].double()], 0)
            z = sum(x[j: j + length] * weight[:, j].double() for j in range(4)) + (0.0 if b is None else b.double())
            want = z * torch.sigmoid(z)
            assert ((out[at: at + length].double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -20 * z.abs() + 1e-7).all()
            at += length


@pytest.mark.parametrize("lens,channels", [([64], 1024), ([255, 3, 1], 1024), ([1] * 65, 1536), ([9, 300, 1], 2048), ([3, 15], 6144),
                                           ([1000, 1, 2, 997, 50], 2048), ([301, 1, 350], 6152)])
def test_short_convolution_has_the_bits_of_the_general_kernel(lens, channels):
    """Rows whose length is no multiple of eight take the general kernel: the same numbers in such rows give the same bits, with one token a
    thread and (from four million sums on) with eight."""
    from edgerag_b200.ops import kernels

    n, off = sum(lens), 16
    g = torch.Generator().manual_seed(n)
    proj = torch.randn(n, channels + 28, generator=g).to(torch.bfloat16).cuda()
    weight, bias = torch.randn(channels, 4, generator=g).to(torch.bfloat16).cuda(), torch.randn(channels, generator=g).to(torch.bfloat16).cuda()
    record = torch.randn(len(lens), 3, channels, generator=g).cuda()
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda()
    seq = torch.tensor([s for s, length in enumerate(lens) for _ in range(length)], dtype=torch.int32).cuda()
    held = torch.arange(len(lens), dtype=torch.int32).cuda()
    for b in (bias, None):
        outs = [torch.empty(n, channels, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        for rows, out in zip((proj[:, : channels + 24].contiguous(), proj), outs):
            kernels.conv_silu(rows, off, weight, b, record, seq, starts, held, out)
        assert torch.equal(*outs)


@pytest.mark.parametrize("n,parts,per", [(1, 1, 128), (5, 3, 256), (33, 2, 512), (3, 1, 1024)])
@pytest.mark.parametrize("gated", [False, True])
def test_group_norm_by_warps(n, parts, per, gated):
    """Against float64: float arithmetic (sums of up to 1,024 squares, 2^-20) rounded once to bfloat16 (2^-8 of the value)."""
    from edgerag_b200.ops import kernels

    g = torch.Generator().manual_seed(per)
    width = parts * per
    x, weight = torch.randn(n, width + 4, generator=g).cuda()[:, :width], torch.randn(width, generator=g).cuda()
    z = torch.randn(n, width + 4, generator=g).to(torch.bfloat16).cuda()[:, 4:] if gated else None
    out = torch.empty(n, width, dtype=torch.bfloat16, device="cuda")
    kernels.gated_group_norm(x, weight, out, 1e-5, parts, gate=z)
    v = x.double() if z is None else x.double() * z.double() * torch.sigmoid(z.double())
    v = v.view(n, parts, per)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(n, width) * weight.double()
    assert ((out.double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -18) + 1e-30).all()


@pytest.mark.parametrize("dv", [4, 124, 128, 132, 256, 512, 6])
def test_head_norm_by_four_values(dv):
    """As above, one weight vector for all heads (6: not in runs of four, the general kernel)."""
    from edgerag_b200.ops import kernels

    g = torch.Generator().manual_seed(dv)
    n, H = 9, 3
    o, weight = torch.randn(n, H * dv, generator=g).cuda(), torch.randn(dv, generator=g).cuda()
    z = torch.randn(n, H * dv + 4, generator=g).to(torch.bfloat16).cuda()[:, : H * dv]
    out = torch.empty(n, H * dv, dtype=torch.bfloat16, device="cuda")
    kernels.head_norm_gate(o, z, weight, out, H, 1e-5)
    v, zz = o.double().view(n, H, dv), z.double().reshape(n, H, dv)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * weight.double() * zz * torch.sigmoid(zz)).view(n, H * dv)
    assert ((out.double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -18) + 1e-30).all()
