"""The cache slots of a prompt portion, worked out page by page.  No GPU."""

import pytest

from tinyvllm_b200.cache.manager import CacheGroup, CacheManager


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9, 40])
@pytest.mark.parametrize("start", [0, 1, 3, 4, 7])
def test_slots_of_a_portion_follow_its_pages(start, count):
    """Token p of a request lies in slot p % page of page table[p // page], wherever the portion starts and ends."""
    manager = CacheManager([CacheGroup((0,), 1, 16)], 4, 32, 2)
    manager.open("other"), manager.open("r")
    for request, n in (("other", 5), ("r", start)):
        if n:
            manager.commit(manager.plan([(request, n)]))
    entry = manager.plan([("r", count)]).entries[0]
    table = entry.tables[0]
    assert entry.slots[0] == tuple(table[p // 4] * 4 + p % 4 for p in range(start, start + count))


def test_a_step_uploads_the_slots_of_its_plan():
    """... of portions and single tokens, in every cache group, with a window whose first pages are given back."""
    from types import SimpleNamespace

    import torch

    from tinyvllm_b200.engine.step import StepEntry, StepRunner

    runner = StepRunner.__new__(StepRunner)
    runner.manager = CacheManager([CacheGroup((0,), 1, 16), CacheGroup((1,), 1, 16, window=6)], 4, [64, 64], 4)
    runner.storage = SimpleNamespace(dtype=torch.float32, clear_state=lambda slots: None)
    runner.tensor_memory_tiles, runner.small_context, runner.cache_sources, runner.max_model_len = False, 0, (), 256
    runner._upload = lambda host, device=None: torch.from_numpy(host.copy())
    for request, held in (("a", 21), ("b", 3), ("c", 0)):
        runner.manager.open(request)
        if held:
            runner.manager.commit(runner.manager.plan([(request, held)]))
    entries = [StepEntry("a", tuple(range(9))), StepEntry("b", (5,)), StepEntry("c", tuple(range(13)))]
    plan = runner.manager.plan([(e.request_id, len(e.tokens)) for e in entries])
    ctx = runner.build_context(entries, plan, split_chunks=0)
    for group in range(2):
        want = []
        for entry in plan.entries:
            table = entry.tables[group]
            want += [table[p // 4] * 4 + p % 4 for p in range(entry.start, entry.start + entry.count)]
        assert ctx.slots[group].tolist() == want
        assert [s for entry in plan.entries for s in entry.slots[group]] == want
