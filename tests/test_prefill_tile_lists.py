"""How a step's prompt entries are cut for the 128-row and the 64-row kernel.  No GPU."""

import pytest

from tinyvllm_b200.ops import kernels
from tinyvllm_b200.ops.attention import prefill_tiles


@pytest.fixture(autouse=True)
def sizes(monkeypatch):
    monkeypatch.setattr(kernels, "attention_prefill_tile_tokens", lambda: 64)
    monkeypatch.setattr(kernels, "attention_prefill_tc_tile_tokens", lambda: 128)


def test_short_rests_and_entries_join_the_tiles_of_a_step_that_has_some():
    big, rest, runs = prefill_tiles([140, 1, 9, 1], [0, 700, 300, 5], tensor_memory=True, singles_apart=True)
    assert big == ([2, 0, 0], [141, 128, 0], [9, 12, 128])              # the longest context first
    assert rest == ([], [], []) and runs == ((140, 1), (150, 1))


def test_a_step_of_short_entries_asks_for_no_tiles():
    assert prefill_tiles([9, 31], [300, 0], tensor_memory=True, singles_apart=True) == (
        ([], [], []), ([], [], []), ((0, 40),))


@pytest.mark.parametrize("counts,starts,small", [([40, 20], [0, 0], True), ([40, 1], [24, 900], True), ([40], [25], False),
                                                 ([9, 65], [0, 0], False)])
def test_small_contexts_stay_with_the_64_row_kernel(counts, starts, small):
    big, rest, _ = prefill_tiles(counts, starts, tensor_memory=True, singles_apart=True, small_context=64)
    assert (len(big[0]) == 0) == small and (len(rest[0]) > 0) == small
