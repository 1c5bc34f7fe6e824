"""The recurrent scans over short portions beside single tokens: the kernel for portions of up to 64 tokens, and blocks for portions alone."""

from __future__ import annotations

import pytest
import torch

from edgerag_b200.ops import kernels
from test_scan_chunks import _delta_reference, _ssm_reference

pytestmark = pytest.mark.gpu


def _error(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("N", [32, 64, 128])
@pytest.mark.parametrize("lens,longest", [([20], 20), ([63], 63), ([64], 64), ([17, 1, 64, 2], 64), ([1] * 40 + [33], 33), ([65, 1, 200], 64)])
def test_state_space_portions_of_up_to_64_tokens(N, lens, longest):
    """Against float64 and beside the walk, with requests behind one another and, by a wrong hint, more than one chunk of 64.  A result is
    off by a few roundings of 24 bits; operands in two pieces instead of three would be off by some 2^-18."""
    H, P, G, n, m = 4, 64, 2, sum(lens), len(lens)
    inner = H * P
    g = torch.Generator().manual_seed(N + n)
    xbc = (torch.randn(n, inner + 2 * G * N, generator=g) * 0.5).to(torch.bfloat16).cuda()
    proj, a_log = torch.randn(n, H, generator=g).to(torch.bfloat16).cuda(), (torch.randn(H, generator=g) * 0.3).cuda()
    dt_bias, skip = torch.randn(H, generator=g).cuda() - 1.0, torch.randn(H, generator=g).cuda()
    before = torch.randn(m, H, N, P, generator=g).cuda()
    starts, slots = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda(), torch.arange(m, dtype=torch.int32).cuda()
    results = []
    for hint, portions in ((longest, 0), (longest, sum(x > 1 for x in lens)), (1, 0)):
        state, y = before.clone(), torch.full((n, inner), float("nan"), device="cuda")
        kernels.ssm_scan(xbc, proj, 0, dt_bias, a_log, skip, state, m, starts, slots, y, G, longest=hint, portions=portions)
        results.append((y, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    assert not torch.equal(results[0][0], results[2][0])
    for s, length in enumerate(lens):
        rows = slice(int(starts[s]), int(starts[s + 1]))
        want_y, want_s = _ssm_reference(xbc[rows], proj[rows], dt_bias, a_log, skip, before[s], H, P, N, G)
        for y, state in results:
            assert _error(y[rows], want_y) < 6e-7 and _error(state[s], want_s) < 6e-7, (s, length)


@pytest.mark.parametrize("lens", [[1] * 40 + [70], [130, 1, 1, 64, 1], [100] * 3, [0] * 20 + [63, 65, 0, 65, 0]])
@pytest.mark.parametrize("scan", ["ssm", "delta"])
def test_blocks_for_portions_alone(scan, lens):
    """Single tokens get no block of the kernels for portions where the caller counts the portions: the same bits."""
    n, m, g = sum(lens), len(lens), torch.Generator().manual_seed(3)
    starts, slots = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32).cuda(), torch.arange(m, dtype=torch.int32).cuda()
    v = [torch.randn(4, generator=g).cuda() - 1.0 for _ in range(3)]
    proj = torch.randn(n, 8, generator=g).to(torch.bfloat16).cuda()
    rows = (torch.randn(n, 4 * 64 + 2 * 2 * 64, generator=g) * 0.5).to(torch.bfloat16).cuda()
    before, outs = 0.3 * torch.randn(m, 4, 64, 64, generator=g).cuda(), []
    for portions in (0, sum(x > 1 for x in lens)):            # (a request may bring no token at all)
        state, out = before.clone(), torch.full((n, 256), float("nan"), device="cuda")
        if scan == "ssm":
            kernels.ssm_scan(rows, proj[:, :4], 0, *v, state, m, starts, slots, out, 2, longest=1 << 20, portions=portions)
        else:
            kernels.delta_scan(rows, proj, 0, 4, v[0], v[1], state, m, starts, slots, out, 2, 64, longest=1 << 20, portions=portions)
        outs.append((out, state))
    assert torch.isfinite(outs[0][0]).all() and all(torch.equal(a, b) for a, b in zip(*outs))
    s = max(range(m), key=lambda i: lens[i])
    at = slice(int(starts[s]), int(starts[s + 1]))
    if scan == "ssm":
        want, want_s = _ssm_reference(rows[at], proj[at, :4], *v, before[s], 4, 64, 64, 2)
    else:
        want, want_s = _delta_reference(rows[at], proj[at, :4], proj[at, 4:], v[0], v[1], before[s], 4, 2, 64, 64)
    assert _error(outs[0][0][at], want) < 8e-7 and _error(outs[0][1][s], want_s) < 8e-7
