"""Which kernel takes single tokens of one query head per kv head (CPU: the launch is recorded, not made)."""

from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels


@pytest.mark.parametrize("how,expected", [({}, 0), ({"window": 512}, 0), ({"softcap": 30.0}, 0), ({"even": True}, 1), ({"tensor_cores": True}, 2),
                                          ({"even": True, "tensor_cores": False}, 0)])
def test_a_launch_says_which_kernel(monkeypatch, how, expected):
    """Masks and shaped scores, which the kernel on CUDA cores makes faster, do not go to the tensor cores by themselves."""
    seen = []
    for name, stand_in in (("_need", lambda *a, **k: None), ("_fn", lambda *a: a), ("_stream", lambda: "stream"), ("split_counters", lambda *a: None),
                           ("_call", lambda fn, *args: seen.append(args))):
        monkeypatch.setattr(kernels, name, stand_in)
    q, pages, i32 = torch.empty(2, 256), torch.empty(9, 4, 16, 64), torch.empty(2, 4, dtype=torch.int32)
    kernels.attention_decode_bulk(q, pages, pages, i32, i32[:, 0], i32[:, 0], q, 4, 0.125, torch.empty(4096), torch.empty(64), 4, i32, split_keys=64, **how)
    assert seen[0][-2:] == (expected, "stream")


@pytest.mark.parametrize("plan,n_seqs,heads,bound,shaped,wanted", [
    ((4096, 2, 2), 8, 32, 8192, False, True), ((8192, 8, 1), 64, 32, 8192, True, True), ((512, 2, 16), 1, 32, 8192, False, True),
    ((128, 2, 48), 1, 8, 5120, False, False), ((768, 2, 1), 8, 32, 768, False, True), ((768, 2, 1), 8, 32, 768, True, False),
    ((256, 2, 1), 8, 32, 256, False, False), ((768, 2, 1), 16, 32, 768, False, False), ((1024, 2, 2), 8, 32, 2048, False, False),
    ((1024, 8, 1), 64, 32, 1024, False, True), ((1024, 4, 1), 32, 32, 1024, False, False), ((768, 8, 1), 64, 32, 768, False, False)])
def test_where_the_tensor_cores_pay(plan, n_seqs, heads, bound, shaped, wanted):
    assert kernels.single_heads_on_tensor_cores(plan, n_seqs, heads, bound, shaped, 148) is wanted


def test_long_pages_keep_single_heads(monkeypatch):
    """Pages of 64 tokens make long copies of one head: short contexts keep the plan that takes them."""
    monkeypatch.setitem(kernels._sm_counts, 0, 148)
    monkeypatch.setattr(kernels.native, "load", lambda *a: SimpleNamespace(erb_attention_decode_even_supported=lambda *a: 1))
    assert kernels._choose_even_plan.__wrapped__(0, 8, 32, 32, 768, 64, 64) is None
    assert kernels._choose_even_plan.__wrapped__(0, 8, 32, 32, 768, 16, 64) == (768, 2, 1)
