"""What a dropped runner leaves behind."""

import gc
import weakref

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
def test_a_dropped_runner_gives_its_memory_back_without_a_collection(model_folders, graphs):
    from edgerag_b200.engine.engine import Engine, EngineOptions
    from edgerag_b200.engine.step import ModelRunner, StepEntry

    folder = model_folders("a", "bfloat16")
    engine = Engine.from_pretrained(folder, EngineOptions(dtype="bfloat16", num_blocks=32, max_batch_size=2))
    gc.collect()
    gc.disable()
    try:
        for turn in range(2):                               # (what the process keeps for good is there after the first)
            before = torch.cuda.memory_allocated()
            runner = ModelRunner(engine.model, engine.cache, engine.pools, max_step_tokens=64, cuda_graphs=graphs)
            for r in range(3):
                runner.admit(r)
                runner.step([StepEntry(r, tokens=[1, 2, 3, 4, 5], want=[4])])
                runner.release(r)
            torch.cuda.synchronize()
            assert runner.graph_replays == (1 if graphs else 0) and torch.cuda.memory_allocated() > before
            dead = weakref.ref(runner)
            del runner
            assert dead() is None
        assert torch.cuda.memory_allocated() == before
    finally:
        gc.enable()
