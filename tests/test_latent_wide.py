"""The form of latent attention that up-projects a portion's context: which sizes take it (CPU)."""

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
