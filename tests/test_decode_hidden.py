"""Decode attention of single tokens: what a token does not see changes no bit of its result; scratch at any float."""

from __future__ import annotations

import pytest
import torch

from edgerag_b200.ops import kernels as K
from test_kernels import paged_case

pytestmark = pytest.mark.gpu


def _run(case, nq, nkv, splits, split, window=0, chunk=0, keep_first=0, heads=0, offset=0, tensor_cores=True):
    dev = {n: case[n].cuda() for n in ("q", "kp", "vp", "tables", "pos")}
    n, d = case["pos"].numel(), case["kp"].shape[3]
    acc, ml = K.decode_scratch_floats(n, nq, d, splits)
    part_acc, part_ml = torch.full((acc,), float("nan"), device="cuda"), torch.full((ml + offset,), float("nan"), device="cuda")[offset:]
    out = torch.full((n, nq * d), float("nan"), dtype=torch.bfloat16, device="cuda")
    status, tok = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")
    args = (dev["q"], dev["kp"], dev["vp"], dev["tables"], tok, dev["pos"], out, nq, d ** -0.5, part_acc, part_ml, splits, status)
    more = {"split_keys": split, "window": window, "chunk": chunk, "keep_first": keep_first}
    if nq == nkv:
        K.attention_decode_bulk(*args, head_group=heads, tensor_cores=tensor_cores, **more)
    else:
        K.attention_decode_gqa(*args, **more)
    torch.cuda.synchronize()
    assert int(status) == 0
    return out.cpu()


@pytest.mark.parametrize("nq,nkv,heads,tensor_cores", [(4, 4, 2, True), (4, 4, 1, True), (4, 4, 2, False), (6, 2, 0, True)])
@pytest.mark.parametrize("mask", [{"window": 37}, {"window": 37, "keep_first": 5}, {"chunk": 24}])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_value_before_the_window_is_not_seen(nq, nkv, heads, tensor_cores, mask, bad):
    """The window (or run) starts inside a page, whose earlier values hold numbers that are not finite."""
    ctx_lens = [60, 131, 40, 200]
    case = paged_case(torch.bfloat16, 5, nq, nkv, 64, 16, ctx_lens, [1] * len(ctx_lens))
    clean = _run(case, nq, nkv, 2, 64, heads=heads, tensor_cores=tensor_cores, **mask)
    hidden = 0
    for s, n in enumerate(ctx_lens):
        lo = max(0, n - mask["window"]) if "window" in mask else (n - 1) // mask["chunk"] * mask["chunk"]
        for key in range(max(lo // 16 * 16, mask.get("keep_first", 0)), lo):
            case["vp"][int(case["tables"][s, key // 16]), :, key % 16] = bad
            hidden += 1
    assert hidden > 8 and torch.isfinite(clean.float()).all()
    assert torch.equal(_run(case, nq, nkv, 2, 64, heads=heads, tensor_cores=tensor_cores, **mask), clean)


@pytest.mark.parametrize("nq,nkv", [(4, 4), (6, 2)])
def test_scratch_that_starts_at_an_odd_float(nq, nkv):
    """The maxima and sums of the splits may lie at any float; partial results that the merge cannot read are refused."""
    case = paged_case(torch.bfloat16, 6, nq, nkv, 64, 16, [60, 200], [1, 1])
    assert torch.equal(_run(case, nq, nkv, 4, 64, offset=1), _run(case, nq, nkv, 4, 64))
    q, pages, i32 = case["q"].cuda(), case["kp"].cuda(), lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")      # noqa: E731
    scratch = torch.zeros(4096, device="cuda")
    call = K.attention_decode_bulk if nq == nkv else K.attention_decode_gqa
    with pytest.raises(K.KernelError, match="aligned"):
        call(q, pages, pages, case["tables"].cuda(), i32(0, 1), case["pos"].cuda(), torch.empty_like(q), nq, 0.125, scratch[1:], scratch, 4, i32(0),
             split_keys=64)
