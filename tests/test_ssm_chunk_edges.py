"""The state-space recurrence 128 tokens at a time, at the edges of its chunks and of the next request's rows."""

import pytest
import torch

from edgerag_b200.ops import kernels
from test_scan_chunks import _ssm_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [32, 64, 128])
@pytest.mark.parametrize("lens", [[127], [128], [129, 1], [256, 255, 2], [257, 5]])
@pytest.mark.parametrize("bad", [False, True])
def test_chunks_of_128_tokens(N, lens, bad):
    """Against float64, within a few hundred roundings of the largest result (both are float throughout), and in the mean within a few: three
    pieces of 8 bits lose nothing, two would leave 2^-18 of every operand, 2e-6 in the mean.  ``bad``: the request behind brings numbers that are not
    finite, which lie in the rows that a chunk's copies reach behind their own request."""
    H, P, G, n = 4, 64, 2, sum(lens)
    inner = H * P
    g = torch.Generator().manual_seed(N + n)
    xbc = (torch.randn(n + 3, inner + 2 * G * N, generator=g) * 0.5).to(torch.bfloat16)
    proj, a_log = torch.randn(n + 3, H, generator=g).to(torch.bfloat16), torch.randn(H, generator=g) * 0.3
    dt_bias, skip, before = torch.randn(H, generator=g) - 1.0, torch.randn(H, generator=g), torch.randn(len(lens) + 1, H, N, P, generator=g)
    if bad:
        xbc[n:] = float("inf")
    starts = torch.tensor([0, *torch.tensor(lens + [3]).cumsum(0).tolist()], dtype=torch.int32).cuda()
    slots = torch.arange(len(lens) + 1, dtype=torch.int32).cuda()
    dev = [t.cuda() for t in (xbc, proj, dt_bias, a_log, skip)]
    state, y = before.clone().cuda(), torch.full((n + 3, inner), float("nan"), device="cuda")
    kernels.ssm_scan(dev[0], dev[1], 0, dev[2], dev[3], dev[4], state, len(lens) + 1, starts, slots, y, G, longest=1 << 20)
    at = 0
    for s, length in enumerate(lens):
        rows = slice(at, at + length)
        want_y, want_s = _ssm_reference(dev[0][rows], dev[1][rows], dev[2], dev[3], dev[4], before[s].cuda(), H, P, N, G)
        assert (y[rows].double() - want_y).abs().max() < 3e-5 * max(1.0, want_y.abs().max()), s
        assert (state[s].double() - want_s).abs().max() < 3e-5 * max(1.0, want_s.abs().max()), s
        for got, want in ((y[rows], want_y), (state[s], want_s)):
            assert (got.double() - want).norm() < 6e-7 * want.norm(), s
        at += length
    assert bad or torch.isfinite(y).all()


@pytest.mark.parametrize("offset", [2, 4])
def test_outputs_on_8_bytes_come_from_the_chunks_too(offset):
    """Outputs that chunks of 128 tokens cannot store come from chunks of 64, not from the walk, whose bits these have not."""
    H, P, N, G, n = 4, 64, 64, 2, 300
    inner = H * P
    g = torch.Generator().manual_seed(1)
    xbc = (torch.randn(n, inner + 2 * G * N, generator=g) * 0.5).to(torch.bfloat16).cuda()
    proj, vec = torch.randn(n, H, generator=g).to(torch.bfloat16).cuda(), [torch.randn(H, generator=g).cuda() - 1.0 for _ in range(3)]
    starts, slots = torch.tensor([0, n], dtype=torch.int32).cuda(), torch.zeros(1, dtype=torch.int32).cuda()

    def scan(y, longest):
        state = torch.zeros(1, H, N, P, device="cuda")
        kernels.ssm_scan(xbc, proj, 0, *vec, state, 1, starts, slots, y, G, longest=longest)
        return y, state

    y, state = scan(torch.empty(n, inner, device="cuda"), n)
    off_y, off_state = scan(torch.empty(n * inner + offset, device="cuda")[offset:].view(n, inner), n)
    short_y, short_state = scan(torch.empty_like(y), 64)
    assert torch.equal(off_y, y if offset == 4 else short_y) and torch.equal(off_state, state if offset == 4 else short_state)
    assert not torch.equal(off_y, scan(torch.empty_like(y), 1)[0]) and not torch.equal(y, short_y)
