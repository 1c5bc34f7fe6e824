"""To which word the scans in chunks report a wait that ran out (CPU: the launches are recorded, not made)."""

from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels
from edgerag_b200.parts import delta, ssd
from edgerag_b200.parts.base import LayerCall


@pytest.fixture()
def launched(monkeypatch):
    """The arguments that reach the entry points, while some other runner's word is the one named last."""
    seen = {}
    for name, stand_in in (("_need", lambda *a, **k: None), ("_fn", lambda library, elem, name: name), ("_stream", lambda: "stream"),
                           ("_call", lambda fn, *args: seen.__setitem__(fn, args)), ("_status_word", "another runner's word")):
        monkeypatch.setattr(kernels, name, stand_in)
    for module in (ssd, delta):
        monkeypatch.setattr(module, "kernels", SimpleNamespace(**{
            **vars(kernels), "linear_parts_count": lambda *a: 0, **{n: lambda *a, **k: None for n in (
                "linear", "conv_silu", "conv_state_update", "gated_group_norm", "head_norm_gate")}}))
    return seen


@pytest.mark.parametrize("word", [None, "this step's word"])
def test_a_part_reports_to_the_word_of_its_step(launched, word):
    cpu, lens = torch.device("cpu"), [40, 1]
    states = {"conv": torch.empty(0), "ssm": torch.empty(2, 4, 64, 32), "delta": torch.empty(2, 4, 32, 64)}
    ctx = SimpleNamespace(batch_invariant=False, host_q_len=lens, n_seqs=2, seq_of_token=None, seq_starts=torch.empty(3), state_slots=torch.empty(2),
                          state=lambda name, layer: states[name], buf=lambda name, shape, dtype: torch.empty(shape, dtype=dtype), status=word)
    for mixer, entry in ((ssd.StateSpaceDuality(64, 4, 32, 64, 2, 4, 2, 1e-5, torch.bfloat16, cpu), "erb_ssm_scan"),
                         (delta.GatedDeltaRule(64, 4, 2, 64, 32, 4, 1e-6, torch.bfloat16, cpu), "erb_delta_scan")):
        for name in ("dt_bias", "a_log", "d_skip"):
            setattr(mixer, name, torch.empty(4))
        mixer.forward(torch.empty(41, 64, dtype=torch.bfloat16), ctx, LayerCall(0, 0))
        assert launched[entry][-2:] == (word, "stream")
