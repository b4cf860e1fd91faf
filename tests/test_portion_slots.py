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
