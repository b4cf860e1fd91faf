"""How a step's prompt entries are cut for the 128-row and the 64-row kernel.  No GPU."""

import pytest

from tinyvllm_b200.ops import kernels
from tinyvllm_b200.ops.attention import prefill_tiles


@pytest.fixture(autouse=True)
def sizes(monkeypatch):
    monkeypatch.setattr(kernels, "attention_prefill_tile_tokens", lambda: 64)
    monkeypatch.setattr(kernels, "attention_prefill_tc_tile_tokens", lambda: 128)


def test_short_rests_are_attended_one_by_one():
    big, rest, runs = prefill_tiles([140, 1, 9, 1], [0, 700, 300, 5], tensor_memory=True, singles_apart=True)
    assert big == ([0], [0], [128])
    assert rest == ([], [], []) and runs == ((128, 23),)


def test_a_step_of_short_entries_asks_for_no_tiles():
    assert prefill_tiles([9, 31], [300, 0], tensor_memory=True, singles_apart=True) == (
        ([], [], []), ([], [], []), ((0, 40),))


@pytest.mark.parametrize("counts,starts,big_rows,rest_rows", [
    ([40, 20], [0, 0], [], [0, 1]), ([40, 1], [24, 900], [], [0]), ([40], [25], [0], []), ([9, 65], [0, 0], [1], [0]),
    ([300, 31, 32], [0, 900, 900], [2, 0, 0, 0], [1])])
def test_entries_go_whole_to_one_of_the_two_kernels(counts, starts, big_rows, rest_rows):
    big, rest, runs = prefill_tiles(counts, starts, tensor_memory=True, singles_apart=True, small_context=64)
    assert (big[0], rest[0]) == (big_rows, rest_rows)
    assert sum(big[2]) + sum(rest[2]) == sum(counts) - counts.count(1) == sum(counts) - sum(n for _, n in runs)


def cut_of(row, counts, starts, small_context):
    """What becomes of entry ``row``: (kernel, first token within the entry, tokens) of every piece, token by token where
    tokens go one by one."""
    big, rest, runs = prefill_tiles(counts, starts, tensor_memory=True, singles_apart=True, small_context=small_context)
    at = sum(counts[:row])
    pieces = [(kind, first - at, count) for kind, lists in (("128", big), ("64", rest))
              for r, first, count in zip(*lists) if r == row]
    for first, count in runs:
        pieces += [("one", t - at, 1) for t in range(max(first, at), min(first + count, at + counts[row]))]
    return sorted(pieces)


@pytest.mark.parametrize("small_context", [0, 64])
@pytest.mark.parametrize("count,start", [(1, 0), (1, 500), (2, 0), (9, 300), (31, 0), (32, 0), (40, 24), (40, 25), (140, 0), (160, 700)])
def test_an_entry_is_cut_the_same_beside_any_other(count, start, small_context):
    alone = cut_of(0, [count], [start], small_context)
    assert sum(n for _, _, n in alone) == count
    for other, at in ((1, 0), (1, 900), (9, 0), (31, 40), (33, 0), (40, 24), (500, 0), (500, 800)):
        assert cut_of(0, [count, other], [start, at], small_context) == alone
        assert cut_of(1, [other, count], [at, start], small_context) == alone
        assert cut_of(1, [other, count, other], [at, start, at], small_context) == alone


def test_asking_whether_windowed_attention_takes_tiles_loads_no_library(monkeypatch):
    from types import SimpleNamespace

    from tinyvllm_b200.ops.attention import windowed_takes_tensor_memory_tiles

    def loaded(name):
        raise AssertionError(f"{name} was loaded")

    monkeypatch.setattr(kernels, "load_library", loaded)
    monkeypatch.setattr(kernels, "_functions", {})
    mixer = SimpleNamespace(key_dim=128, value_dim=128, softcap=None, distance_slope_exponent=None, segment=1024, window=None,
                            distance_table=(32, 1024.0), num_heads=16, num_kv_heads=8)
    assert windowed_takes_tensor_memory_tiles(mixer, 16)
    mixer.distance_table = (32, float(kernels.PREFILL_TC_BIAS_ROWS))
    assert not windowed_takes_tensor_memory_tiles(mixer, 16)


def test_the_library_takes_as_long_a_bias_as_it_is_said_to():
    assert kernels._fn("attention_prefill_tc", "tvb_attention_prefill_tc_bias_rows", [])() == kernels.PREFILL_TC_BIAS_ROWS
