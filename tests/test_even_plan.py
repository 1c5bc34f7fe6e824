"""The plan of equal splits at long contexts (CPU: what the library answers is stood in for)."""

from types import SimpleNamespace

import pytest

from edgerag_b200.ops import kernels


@pytest.mark.parametrize("n_seqs,nq,nkv,bound,page", [(200, 15, 5, 1 << 20, 16), (200, 15, 5, 1 << 18, 8), (200, 4, 1, 400_000, 16), (30, 8, 8, 1 << 21, 16),
                                                      (1, 15, 5, 1 << 24, 8), (200, 15, 5, 8192, 16)])
def test_a_split_has_room_for_its_pages(monkeypatch, n_seqs, nq, nkv, bound, page):
    """One wave of blocks cuts few splits of many sequences: they keep to what shared memory holds, or the other plan stands."""
    monkeypatch.setitem(kernels._sm_counts, 0, 148)
    monkeypatch.setattr(kernels.native, "load", lambda *a: SimpleNamespace(erb_attention_decode_bulk_groups=lambda *a: 1,
                                                                           erb_attention_decode_even_supported=lambda *a: 1))
    plan = kernels._choose_even_plan.__wrapped__(0, n_seqs, nq, nkv, bound, page, 64)
    assert plan is None or (plan[0] <= 1024 * page and plan[0] * plan[2] >= bound)
    assert bound > 8192 or plan is not None


@pytest.mark.parametrize("n_seqs,bound,plan", [(1, 256, (48, 0, 6)), (8, 512, (64, 0, 8)), (8, 768, (96, 0, 8)), (8, 1024, (64, 0, 16)), (4, 1536, (64, 0, 24)),
                                               (1, 4096, (128, 0, 32)), (4, 3072, (96, 0, 32)), (2, 8192, None), (8, 8192, (256, 0, 32)), (64, 8192, (2048, 0, 4))])
def test_splits_of_grouped_heads(monkeypatch, n_seqs, bound, plan):
    """No more splits than their merge pays for, whatever a wave would hold."""
    monkeypatch.setitem(kernels._sm_counts, 0, 148)
    monkeypatch.setattr(kernels.native, "load", lambda *a: SimpleNamespace(erb_attention_decode_bulk_groups=lambda *a: 1,
                                                                           erb_attention_decode_even_supported=lambda *a: 1))
    assert kernels._choose_even_plan.__wrapped__(0, n_seqs, 15, 5, bound, 16, 64) == plan
