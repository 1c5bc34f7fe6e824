"""The form of latent attention that up-projects a portion's context: which sizes and steps take it (CPU)."""

from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels


@pytest.mark.parametrize("rank", [8, 64, 512, 520, 576, 640, 960, 1024])
@pytest.mark.parametrize("dim,rot,v", [(64, 8, 64), (64, 32, 128), (128, 64, 128), (128, 64, 64)])
def test_no_size_is_rounded_more_than_in_the_latent_space(dim, rot, v, rank):
    """Where the latent space has float32 queries and weights (the general kernel), the up-projected form is not taken."""
    wide = kernels.latent_wide_supported(torch.bfloat16, dim, rot, v, rank)
    assert wide == (kernels.latent_mma_supported(torch.bfloat16, rank, rot) and rank <= 512)
    assert not kernels.latent_wide_supported(torch.float32, dim, rot, v, rank)


def _mixer(heads, dim, rot, v, rank, **more):
    from edgerag_b200.parts.latent_attention import LatentAttention

    return LatentAttention(64, heads, dim, rot, v, rank, 0.1, 10000.0, rot, 1e-5, torch.bfloat16, torch.device("cpu"), **more)


@pytest.mark.parametrize("mixer,lens,rows,wide", [
    # device times of the sublayer, up-projected | in the latent space
    ((16, 128, 64, 128, 512), [2], 64, True),                         # 25 | 35 us
    ((16, 128, 64, 128, 512), [2], 8192, True),                       # 204 | 645
    ((16, 128, 64, 128, 512), [2, 3, 3, 3], 8192, True),              # 285 | 646
    ((16, 128, 64, 128, 512), [2] * 8, 2048, True),                   # 125 | 189
    ((16, 128, 64, 128, 512), [2] * 16, 2048, False),                 # 187 to 232 | 189 to 191
    ((16, 128, 64, 128, 512), [2] * 16, 512, False),                  # 96 | 74
    ((16, 128, 64, 128, 512), [2] * 32, 1024, False),                 # 186 | 113
    ((16, 128, 64, 128, 512), [2] * 32, 64, False),                   # 62 | 41
    ((16, 128, 64, 128, 512), [512] + [17] * 15, 2048, True),         # 205 | 350
    ((16, 128, 64, 128, 512), [512] + [17] * 15, 512, True),          # 99 | 119
    ((16, 128, 64, 128, 512), [1531, 517], 1536, True),
    ((8, 64, 32, 64, 256), [2], 64, True),                            # 21 | 23
    ((8, 64, 32, 64, 256), [2] * 16, 2048, True),                     # 74 | 133
    ((8, 64, 32, 64, 256), [2] * 32, 64, False),                      # 34 | 29
])
def test_portions_take_the_faster_form(mixer, lens, rows, wide, monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    step = SimpleNamespace(batch_invariant=False, host_q_len=lens, n_decode=0, max_keys_bound=lambda: rows)
    assert _mixer(*mixer)._wide_rows(step) == (rows if wide else 0)
    # beside single tokens whose contexts set the bound, and where nothing may depend on the step: the latent space
    step.host_q_len, step.n_decode = [1] * 8 + lens, 8
    if rows * len(lens) > 32 * sum(lens) + 2048:
        assert _mixer(*mixer)._wide_rows(step) == 0
    step.batch_invariant = True
    assert _mixer(*mixer)._wide_rows(step) == 0


def test_rows_follow_the_window_and_the_limit_of_bytes(monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    step = SimpleNamespace(batch_invariant=False, host_q_len=[100], n_decode=0, max_keys_bound=lambda: 4096)
    mixer = _mixer(16, 128, 64, 128, 512, window=200)
    assert mixer._wide_rows(step) == 384                              # 200 + 100 + 63 keys, whole tiles of 64
    mixer.WIDE_MAX_BYTES = 2 * 384 * 16 * 256 - 1
    assert mixer._wide_rows(step) == 0
