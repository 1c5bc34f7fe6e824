"""Decode attention whose sequences are cut into equally many splits each, and the tensor-core kernel with one query head per kv head
(its weights in three pieces): against the reference, over the edges of pages, splits and stages."""

from __future__ import annotations

import pytest
import torch

from edgerag_b200.ops import kernels as K
from test_kernels import attention_reference, paged_case, tol

pytestmark = pytest.mark.gpu


def _run(case, nq, nkv, d, splits, split, heads, even=True, parts=False):
    dev = {n: case[n].cuda() for n in ("q", "kp", "vp", "tables", "pos")}
    n = case["pos"].numel()
    acc, ml = K.decode_scratch_floats(n, nq, d, splits)
    part_acc, part_ml = (torch.full((m,), float("nan"), device="cuda") for m in (acc, ml))
    out = torch.full((n, nq * d), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tok = torch.arange(n, dtype=torch.int32, device="cuda")
    args = (dev["q"], dev["kp"], dev["vp"], dev["tables"], tok, dev["pos"], out, nq, d ** -0.5, part_acc, part_ml, splits, status)
    if nq == nkv:
        K.attention_decode_bulk(*args, split_keys=split, head_group=heads, even=even)
    else:
        K.attention_decode_gqa(*args, split_keys=split, even=even)
    torch.cuda.synchronize()
    assert int(status) == 0 and int(K.split_counters(out.device, 1).abs().sum()) == 0
    return (part_acc.view(n, nq, splits, d).cpu(), part_ml.view(n, nq, splits, 2).cpu()) if parts else out


def _of_the_parts(case, nq, nkv, parts):
    """The splits' partial results put together in 64 bits, and the same attention in 64 bits."""
    acc, ml = (p.double() for p in parts)
    there = ~ml[..., 0].isnan()
    top = torch.where(there, ml[..., 0], -torch.inf)
    w = torch.exp2(top - top.amax(-1, keepdim=True))
    got = (torch.where(there[..., None], acc, 0.0) * w[..., None]).sum(2) / (torch.where(there, ml[..., 1], 0.0) * w).sum(-1, keepdim=True)
    want = []
    for t in range(acc.shape[0]):
        k, v = (x[t].double().repeat_interleave(nq // nkv, 1) for x in (case["ks"], case["vs"]))
        score = torch.einsum("hd,khd->hk", case["q"][t].double().view(nq, -1), k) * 0.125
        want.append(torch.einsum("hk,khd->hd", torch.softmax(score, -1), v))
    return got, torch.stack(want)


@pytest.mark.parametrize("nq,nkv,heads", [(8, 8, 2), (5, 5, 4), (9, 9, 8), (4, 4, 1), (15, 5, 0), (6, 3, 0)])
@pytest.mark.parametrize("splits", [2, 7])
def test_the_parts_of_equal_splits(nq, nkv, heads, splits):
    """Every sequence is cut into as many whole pages as its own length gives, not at multiples of the longest's.  One query head per kv head: a
    weight goes in whole, as three pieces; rounded to 16 bits, weights of several query heads among them, it is off by 2^-9, in two by 2^-18."""
    ctx_lens = [17, 129, 500, 1300]
    case = paged_case(torch.bfloat16, 11 + splits, nq, nkv, 64, 16, ctx_lens, [1] * len(ctx_lens))
    parts = _run(case, nq, nkv, 64, splits, -(-max(ctx_lens) // (splits * 16)) * 16, heads, parts=True)
    written = [-(-n // (-(-n // (splits * 16)) * 16)) for n in ctx_lens]
    assert (~parts[1][..., 0].isnan()).sum(-1).tolist() == [[w] * nq for w in written]
    got, want = _of_the_parts(case, nq, nkv, parts)
    assert (got - want).norm() < (6e-7 if nq == nkv else 4e-3) * want.norm()


@pytest.mark.parametrize("nq,nkv,ps,heads", [(8, 8, 16, 2), (5, 5, 16, 4), (9, 9, 8, 8), (3, 3, 128, 1), (15, 5, 16, 0), (6, 3, 64, 0)])
@pytest.mark.parametrize("splits", [1, 2, 7, 64])
def test_equal_splits(nq, nkv, ps, heads, splits):
    ctx_lens = [1, 2, 15, 16, 17, 127, 128, 129, 500, 1300]
    case = paged_case(torch.bfloat16, 7 + ps + splits, nq, nkv, 64, ps, ctx_lens, [1] * len(ctx_lens))
    most = -(-max(ctx_lens) // (splits * ps)) * ps
    got = _run(case, nq, nkv, 64, splits, most, heads)
    torch.testing.assert_close(got.float().cpu(), attention_reference(case, nq, nkv, 64, 0.125), **tol(torch.bfloat16))


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_a_value_that_is_not_finite_stays_in_its_entry(bad):
    """One query head per kv head: an infinity in the values gives an infinity (the pieces of its weight do not cancel), elsewhere nothing changes."""
    case = paged_case(torch.bfloat16, 3, 4, 4, 64, 16, [200], [1])
    clean = _run(case, 4, 4, 64, 3, 80, 2).float().cpu()
    row = int(case["tables"][0, 2])
    case["vp"][row, 1, 5, 9] = bad
    got = _run(case, 4, 4, 64, 3, 80, 2).float().cpu()
    at = 1 * 64 + 9
    assert torch.equal(torch.isfinite(got[0]), torch.arange(256) != at)
    assert torch.equal(got[0, at], torch.tensor(bad)) or bad != bad
    keep = torch.arange(256) != at
    assert torch.equal(got[0, keep], clean[0, keep])


@pytest.mark.parametrize("nq,nkv", [(32, 32), (15, 5), (9, 3), (6, 6)])
def test_the_plan_of_equal_splits(nq, nkv):
    """Never more than one wave of blocks or 64 splits, whole pages, the bound covered; nothing for sizes that the kernel does not take."""
    slots = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (1, 3, 8, 17, 64, 200, 1000):
        for bound in (16, 128, 384, 768, 8192, 65536):
            plan = K.choose_even_plan(n, nq, nkv, bound, 16, 64)
            if plan is not None:
                split, heads, splits = plan
                groups = -(-nkv // (heads or 8))
                assert split % 16 == 0 and split * splits >= bound and splits <= 64 and n * groups * splits <= slots
    assert K.choose_even_plan(8, nq, nkv, 1024, 16, 128) is None and K.choose_even_plan(8, nq, nkv, 1024, 12, 64) is None
    assert K.choose_even_plan(8, nq, nkv, 8192, 16, 64) is not None and K.choose_even_plan(64, nq, nkv, 8192, 16, 64) is not None


@pytest.mark.parametrize("batch,nq,nkv,context,kernel,equal", [(64, 15, 5, 700, "gqa", True), (8, 32, 32, 1000, "bulk", False), (8, 32, 32, 2500, "bulk", True)])
def test_the_timed_launch_is_the_engines(batch, nq, nkv, context, kernel, equal):
    """The program that times one kernel takes the splits that a step of these sequences takes."""
    from argparse import Namespace

    from edgerag_b200.ops import microbench

    a = Namespace(batch=batch, context=context, heads=nq, kv_heads=nkv, head_dim=64, page=16, split=0, kernel=kernel, head_group=0, dtype="bfloat16",
                  cold=False, iters=2, warmup=1, sequential_pages=False)
    out = microbench.decode_attention(a)
    split, heads, splits = K.choose_even_plan(batch, nq, nkv, K.context_bound(-(-context // 16))[0] * 16, 16, 64)
    assert (out["split"], out["head_group"], out["splits"], out["even"], out["status"]) == (split, heads, splits, equal, 0)
