"""What ``batch_invariant`` pins in the mixers whose kernels are chosen by the whole step (CPU: the kernels are recorded, not run)."""

from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels
from edgerag_b200.parts import delta, ssd
from edgerag_b200.parts.base import LayerCall
from edgerag_b200.parts.diff_attention import DiffAttention


class Recorder:
    """Stands in for the module of kernels: launches are recorded, everything else is the module's own."""

    LAUNCHES = ("linear", "conv_silu", "conv_state_update", "ssm_scan", "delta_scan", "gated_group_norm", "head_norm_gate")

    def __init__(self):
        self.calls = {}

    def __getattr__(self, name):
        if name == "linear_parts_count":
            return lambda *a: 0
        if name in self.LAUNCHES:
            return lambda *a, **k: self.calls.__setitem__(name, (a, k))
        return getattr(kernels, name)


def step(lens, batch_invariant):
    return SimpleNamespace(batch_invariant=batch_invariant, host_q_len=lens, n_seqs=len(lens), n_decode=sum(n == 1 for n in lens), page_size=16,
                           seq_of_token=None, seq_starts=None, state_slots=None, state=lambda name, layer: None,
                           max_keys_bound=lambda: 4096, buf=lambda name, shape, dtype: torch.empty(shape, dtype=dtype))


@pytest.mark.parametrize("lens", [[30], [1, 30], [30] + [8] * 31, [500, 64]])
def test_scans_walk_every_token(lens, monkeypatch):
    cpu, n = torch.device("cpu"), sum(lens)
    mixers = {ssd: (ssd.StateSpaceDuality(64, 4, 32, 64, 2, 4, 2, 1e-5, torch.bfloat16, cpu), "ssm_scan"),
              delta: (delta.GatedDeltaRule(64, 4, 2, 64, 32, 4, 1e-6, torch.bfloat16, cpu), "delta_scan")}
    for module, (mixer, scan) in mixers.items():
        for pinned in (True, False):
            seen = Recorder()
            monkeypatch.setattr(module, "kernels", seen)
            mixer.forward(torch.empty(n, 64, dtype=torch.bfloat16), step(lens, pinned), LayerCall(0, 0))
            args, named = seen.calls[scan]
            assert named["longest"] == (1 if pinned else max(lens))
            if scan == "delta_scan":
                assert args[-1].numel() == kernels.delta_scratch_floats(n, 4, 2, 64, 32, 0 if pinned else len(lens))


def test_differential_portions_keep_their_kernel(monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    mixer = DiffAttention(64, 4, 2, 64, 128, 0.125, 0.4, 1e-5, torch.bfloat16, torch.device("cpu"))
    assert mixer._wide_blocks(step([300], False), 300) == 3
    assert mixer._wide_blocks(step([300], True), 300) == 0
