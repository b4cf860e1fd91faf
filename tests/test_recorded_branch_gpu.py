"""Decoded tokens beside prompt portions run as a branch of a recorded step: the replayed step gives the bits of the eager one."""

import pytest
import torch

from test_engine_gpu import make_runner
from tiny_configs import TINY_CONFIGS, random_tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,page", [("a", 16), ("e", 16), ("f", 8)])
def test_replayed_mixed_steps_equal_eager_ones(model_folders, name, page):
    from tinyvllm_b200.engine.step import StepEntry

    if name not in TINY_CONFIGS:
        pytest.skip("no such configuration")
    vocab = TINY_CONFIGS[name].vocab_size
    eager = make_runner(model_folders[name], torch.bfloat16, page, 64)
    graphed = make_runner(model_folders[name], torch.bfloat16, page, 64)
    graphed.enable_step_graphs(limit=2)
    graphed.CAPTURE_AT_OCCURRENCE, graphed.CAPTURE_EVERY_STEPS, graphed.KEEP_FOR_STEPS = 2, 0, 0
    for turn in range(5):
        rows = []
        for runner in (eager, graphed):
            for request, count in (("a", 70), ("b", 33)):
                runner.open(request)
                runner.run([StepEntry(request, tuple(random_tokens(vocab, count, 10 * turn + count)))])
            runner.open("c")
            entries = [StepEntry("a", (3,), (0,)), StepEntry("b", (4,), (0,)),
                       StepEntry("c", tuple(random_tokens(vocab, 150, turn)), (0, 149))]
            rows.append(runner.run(entries).clone())
            rows.append(runner.run([StepEntry(r, (5,), (0,)) for r in "abc"]).clone())        # what the step left in the cache
            for request in "abc":
                runner.close(request)
        assert torch.equal(rows[0], rows[2]) and torch.equal(rows[1], rows[3]), turn
    assert graphed._step_graphs
