"""The 32-bit attention that takes 32 neighbouring tokens together, against the kernel of single rows and float64: portions whose ends fall
inside a block, several sequences in one block, windows with kept keys, chunks, penalties, caps, gates, both head sizes; and that no value
of a key that a row does not see reaches it."""

from __future__ import annotations

import pytest
import torch

from edgerag_b200.ops import kernels as K


@pytest.mark.gpu
@pytest.mark.parametrize("dim,heads,kv,page,portions,how", [
    (64, 9, 3, 16, ((333, 0),), {}),
    (64, 4, 4, 8, ((31, 0), (1, 5), (33, 64), (2, 191), (65, 130)), {}),
    (128, 4, 2, 12, ((95, 33), (64, 0)), {"gate": True}),
    (64, 4, 1, 32, ((200, 300), (40, 0)), {"window": 70, "keep_first": 3}),
    (64, 2, 2, 16, ((130, 700),), {"window": 33, "keep_first": 129}),
    (128, 2, 1, 16, ((150, 77),), {"chunk": 50}),
    (64, 6, 2, 64, ((128, 64),), {"penalty": True}),
    (64, 3, 3, 16, ((64, 1000), (97, 3)), {"softcap": 2.0}),
])
def test_tokens_together_as_alone(dim, heads, kv, page, portions, how):
    g = torch.Generator().manual_seed(dim + len(portions) + portions[0][0])
    how, n = dict(how), sum(a for a, _ in portions)
    per = max(-(-(a + p) // page) for a, p in portions)
    tables = torch.randperm(per * len(portions), generator=g).view(len(portions), per).int()
    keys, values = (torch.randn(per * len(portions), kv, page, dim, generator=g) for _ in range(2))
    q = torch.randn(n, heads * dim + 24, generator=g)[:, : heads * dim]
    seq = torch.cat([torch.full((a,), i) for i, (a, _) in enumerate(portions)]).int()
    pos = torch.cat([torch.arange(p, p + a) for a, p in portions]).int()
    gate = torch.randn(n, heads * dim, generator=g) if how.pop("gate", False) else None
    penalty = torch.rand(2, heads, generator=g) if how.pop("penalty", False) else None
    window, kept, chunk, cap = (how.get(k, 0) for k in ("window", "keep_first", "chunk", "softcap"))
    scale = dim ** -0.5
    cuda = lambda t: None if t is None else t.cuda()     # noqa: E731
    args = [cuda(t) for t in (q, keys, values, tables, seq, pos)]

    def run(tiled, k=args[1], v=args[2]):
        out = torch.full((n, heads * dim), float("nan"), device="cuda")
        K.attention_rows(args[0], k, v, *args[3:], out, heads, scale, penalty=cuda(penalty), gate=cuda(gate), tiled=tiled, **how)
        return out.cpu()

    together, alone = run(True), run(False)
    want, spread = torch.empty(n, heads * dim, dtype=torch.float64), 0.0
    for t in range(n):
        s, p = int(seq[t]), int(pos[t])
        at = torch.arange(p + 1)
        seen = (at >= p // chunk * chunk) if chunk else ((at > p - window) | (at < kept)) if window else at >= 0
        at = at[seen]
        k, v = (x[tables[s].long()[at // page], :, at % page].double().repeat_interleave(heads // kv, 1) for x in (keys, values))
        qt = q[t].double().view(heads, dim)
        z = torch.einsum("hd,khd->hk", qt, k) * scale
        spread = max(spread, float(torch.einsum("hd,khd->hk", qt.abs(), k.abs()).max()) * scale)
        if penalty is not None:
            z = z - penalty[0].double()[:, None] * torch.log1p(penalty[1].double()[:, None] * (p - at).double())
        if cap:
            z = cap * torch.tanh(z / cap)
        o = torch.einsum("hk,khd->hd", torch.softmax(z, 1), v).reshape(-1)
        want[t] = o if gate is None else o * torch.sigmoid(gate[t].double())
    # a score is off by at most dim + 8 roundings of its products' magnitudes, a weight by twice that (its own and the sum's) and 8 more
    # roundings, the sums over keys by 64 + keys / 64 each; the outputs are averages of values
    e = 2.0 ** -24
    bound = (2 * (dim + 8) * e * spread + (8 + 2 * (64 + int(pos.max()) / 64)) * e) * float(values.abs().max())
    assert (alone.double() - want).abs().max() <= bound
    assert (together.double() - want).abs().max() <= bound
    # rounding of the same size as the row kernel's (both are sums of the same terms; the largest of thousands of errors varies by tens of per cent)
    assert (together.double() - want).pow(2).mean().sqrt() <= 1.25 * (alone.double() - want).pow(2).mean().sqrt()

    # keys after a row's position hold values that are no numbers: no earlier row may notice
    bad = values.clone()
    last = len(portions) - 1
    p_last = int(pos[-1])
    bad[tables[last, p_last // page].long(), :, p_last % page] = float("inf")
    poisoned = run(True, v=bad.cuda())
    assert torch.equal(poisoned[: n - 1], together[: n - 1]) and not torch.isfinite(poisoned[n - 1]).any()
    # and a row does not depend on the tokens beside it
    if portions[0][0] > 40:
        cut = [args[0][17:], args[1], args[2], args[3], args[4][17:], args[5][17:]]
        out = torch.empty(n - 17, heads * dim, device="cuda")
        K.attention_rows(*cut, out, heads, scale, penalty=cuda(penalty), gate=cuda(gate)[17:] if gate is not None else None, tiled=True, **how)
        assert torch.equal(out.cpu(), together[17:])


@pytest.mark.gpu
@pytest.mark.parametrize("how", [{}, {"window": 70, "keep_first": 5}, {"chunk": 100}, {"softcap": 20.0}])
@pytest.mark.parametrize("lens,pasts", [([96], [0]), ([32, 32, 33], [0, 100, 31]), ([200, 7, 65], [300, 0, 64])])
def test_one_group_of_threads_gives_the_bits_of_two(how, lens, pasts):
    """The even and the odd key tiles one after the other or side by side, blocks of one and of several requests."""
    from test_kernels import paged_case

    case = paged_case(torch.float32, 9, 6, 2, 64, 16, [n + p for n, p in zip(lens, pasts)], lens)
    dev = [case[n].cuda() for n in ("q", "kp", "vp", "tables", "seq_of", "pos")]
    outs = []
    for tiled in (1, 2):
        out = torch.full_like(dev[0], float("nan"))
        K.attention_rows(*dev, out, 6, 0.125, tiled=tiled, **how)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)
