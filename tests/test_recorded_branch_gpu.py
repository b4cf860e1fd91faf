"""Decoded tokens beside prompt portions run as a branch of a recorded step: the replayed step gives the bits of the eager one."""

import pytest
import torch

from test_engine_gpu import make_runner
from tiny_configs import TINY_CONFIGS, random_tokens

pytestmark = pytest.mark.gpu


def mixed_step(runner, vocab, turn):
    """The logits of a step of two decoded tokens and a portion, and of a decode step behind it."""
    from tinyvllm_b200.engine.step import StepEntry

    for request, count in (("a", 70), ("b", 33)):
        runner.open(request)
        runner.run([StepEntry(request, tuple(random_tokens(vocab, count, 10 * turn + count)))])
    runner.open("c")
    entries = [StepEntry("a", (3,), (0,)), StepEntry("b", (4,), (0,)),
               StepEntry("c", tuple(random_tokens(vocab, 150, turn)), (0, 149))]
    rows = [runner.run(entries).clone(),
            runner.run([StepEntry(r, (5,), (0,)) for r in "abc"]).clone()]        # what the step left in the cache
    for request in "abc":
        runner.close(request)
    return rows


def watch_attention(monkeypatch, noted):
    """Every attention launch of a step: (the kernel, its stream, whether it is being recorded, rows of q)."""
    from tinyvllm_b200.ops import kernels

    for name in ("attention_decode", "attention_rows", "attention_prefill", "attention_prefill_tc"):
        def watched(q, *args, name=name, launch=getattr(kernels, name), **words):
            noted.append((name, torch.cuda.current_stream().cuda_stream, torch.cuda.is_current_stream_capturing(), q.shape[0]))
            return launch(q, *args, **words)
        monkeypatch.setattr(kernels, name, watched)


def recording(runner):
    runner.enable_step_graphs(limit=2)
    runner.CAPTURE_AT_OCCURRENCE, runner.CAPTURE_EVERY_STEPS, runner.KEEP_FOR_STEPS = 2, 0, 0
    return runner


# (d: heads of 64 and a window, e: heads of 128: both take the tile kernels and the decode kernel)
@pytest.mark.parametrize("name,page", [("d", 16), ("e", 16)])
def test_replayed_mixed_steps_equal_eager_ones(model_folders, monkeypatch, name, page):
    vocab, layers = TINY_CONFIGS[name].vocab_size, TINY_CONFIGS[name].num_hidden_layers
    eager = make_runner(model_folders[name], torch.bfloat16, page, 64)
    graphed = recording(make_runner(model_folders[name], torch.bfloat16, page, 64))
    noted = []
    watch_attention(monkeypatch, noted)
    for turn in range(5):
        noted.clear()
        want = mixed_step(eager, vocab, turn)
        # eager: one stream, the tiles of a layer before its single tokens
        of_mixed = [at for at, (kernel, _, _, _) in enumerate(noted) if kernel.startswith("attention_prefill")][-layers:]
        singles = [at for at, (kernel, _, _, rows) in enumerate(noted) if kernel in ("attention_decode", "attention_rows") and rows == 2]
        assert len(of_mixed) == len(singles) == layers and all(tile < single for tile, single in zip(of_mixed, singles))
        assert len({stream for _, stream, _, _ in noted}) == 1 and not any(captured for _, _, captured, _ in noted)
        noted.clear()
        got = mixed_step(graphed, vocab, turn)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), turn
        if turn == 1:
            # recorded: single tokens on a stream beside the tiles'
            streams = {kind: {stream for kernel, stream, captured, rows in noted
                              if captured and kernel.startswith("attention_prefill") == (kind == "tiles") and rows in (2, 152)}
                       for kind in ("tiles", "singles")}
            assert len(streams["tiles"]) == len(streams["singles"]) == 1 and streams["tiles"] != streams["singles"]
    assert graphed._step_graphs


def test_a_failed_recording_leaves_the_step_on_one_stream(model_folders, monkeypatch):
    runner = recording(make_runner(model_folders["e"], torch.bfloat16, 16, 64))
    vocab, forward, seen = TINY_CONFIGS["e"].vocab_size, runner.model.forward, []

    def fails_while_recorded(ctx):
        if torch.cuda.is_current_stream_capturing():
            seen.append(ctx)
            assert ctx.side_stream is not None
            raise RuntimeError("a part that cannot be recorded")
        assert ctx.side_stream is None
        return forward(ctx)

    want = mixed_step(runner, vocab, 0)
    monkeypatch.setattr(runner.model, "forward", fails_while_recorded)
    for turn in (0, 0):
        got = mixed_step(runner, vocab, turn)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert seen and seen[0].side_stream is None and not runner._step_graphs
