"""The short convolution's silu over every bfloat16 number, one tap of weight 1: against float64 and beside v / (1 + exp(-v)) in float."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [4096, 4100])          # by eight channels (several tokens a thread) and by the general kernel
def test_silu_of_every_bfloat16_number(channels):
    from edgerag_b200.ops import kernels

    every = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    n = 1200
    x = every.repeat(-(-n * channels // 65536))[: n * channels].view(n, channels).cuda()
    weight = torch.zeros(channels, 4, dtype=torch.bfloat16, device="cuda")
    weight[:, 3] = 1.0
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    # (the other taps multiply by 0: every input that is not finite would reach the three tokens behind it, so requests of one token)
    starts, seq = torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")
    out = torch.empty_like(x)
    kernels.conv_silu(x, 0, weight, None, torch.zeros(1, 3, channels, device="cuda"), seq, starts, i32(*[0] * n), out)
    v = x.float() + 0.0
    plain, exact = (v / (1 + torch.exp(-v))).to(torch.bfloat16), v.double() / (1 + torch.exp(-v.double()))
    fine = torch.isfinite(plain) & torch.isfinite(v)
    assert torch.equal(torch.isfinite(out), torch.isfinite(plain)) and torch.equal(torch.isnan(out), torch.isnan(plain))
    # half a unit of the last of bfloat16's 8 bits (2^-8 of the value at most) and the float error before it; below 2^-120 exp(-v) has left
    # float's range
    bound = exact.abs() * (2.0 ** -8 + 2.0 ** -21) + 2.0 ** -120
    assert ((out.double() - exact).abs() <= bound)[fine].all()
    wrong = lambda y: int((y != exact.to(torch.bfloat16))[fine & (v > -80)].sum())      # noqa: E731   (not the nearest bfloat16)
    assert wrong(out) <= wrong(plain) + n * channels // 65536 * 2, (wrong(out), wrong(plain))
