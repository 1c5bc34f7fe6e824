"""Which portions of differential attention the tcgen05 kernel takes (CPU; device times of both kernels beside each case)."""

from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels
from edgerag_b200.parts.diff_attention import DiffAttention


@pytest.mark.parametrize("heads,kv,window,cap,lens,bound,wide", [
    # tcgen05 | 64 rows, us
    (16, 4, 0, 30.0, [2048], 2048, 1),                       # 71 | 240
    (16, 4, 0, 0.0, [33], 1280, 1),                          # 32 | 57
    (16, 4, 0, 0.0, [17] * 32, 64, 0),                       # 36 | 15
    (16, 4, 0, 30.0, [17] * 32, 1024, 0),                    # 149 | 87
    (16, 4, 128, 30.0, [300], 1024, 0),                      # 26 | 21
    (16, 4, 512, 30.0, [300] + [2] * 15, 320, 0),            # 33 | 21
    (16, 4, 0, 30.0, [512] + [17] * 7, 2048, 1),             # 71 | 156
    (8, 2, 0, 30.0, [17] * 32, 64, 0),                       # 22 | 14
    (4, 4, 0, 0.0, [130], 640, 1),
    (16, 4, 0, 30.0, [31], 4096, 0),                         # fewer tokens than the kernels of tiles are for
])
def test_portions_take_the_faster_kernel(heads, kv, window, cap, lens, bound, wide, monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    mixer = DiffAttention(64, heads, kv, 64, 128, 0.125, 0.4, 1e-5, torch.bfloat16, torch.device("cpu"), window=window, softcap=cap)
    step = SimpleNamespace(batch_invariant=False, page_size=16, n_decode=0, host_q_len=lens, max_keys_bound=lambda: bound)
    blocks = sum(-(-n // kernels.DIFF_WIDE_ROWS) for n in lens)
    assert mixer._wide_blocks(step, sum(lens)) == blocks * wide
