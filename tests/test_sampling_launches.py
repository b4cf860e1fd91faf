"""How sampling is launched: how many kernels, and that programmatic launch can be turned off.  No GPU."""

import pytest
import torch

from tinyvllm_b200.ops import kernels


@pytest.fixture
def asked(monkeypatch):
    """The arguments of the calls into the library, which launch nothing here."""
    calls = []

    def recorded(library, name, argtypes, restype=None):
        if name == "tvb_sample_rows":
            return lambda *args: calls.append(args) or 0
        return original(library, name, argtypes)

    original = kernels._fn
    monkeypatch.setattr(kernels, "_fn", recorded)
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    return calls


@pytest.mark.parametrize("switched_on,first,second", [(frozenset(), 0, 0), (frozenset(kernels._PDL_DEFAULT), 0, 1),
                                                      (frozenset({"sample"}), 1, 0), (frozenset({"sample", "sample_second"}), 1, 1)])
@pytest.mark.parametrize("rows,launches", [(1, 1), (37, 1), (38, 2), (64, 2)])
def test_programmatic_launch_follows_the_switch(asked, monkeypatch, switched_on, first, second, rows, launches):
    monkeypatch.setattr(kernels, "PDL", switched_on)
    before = kernels.launch_count()
    kernels.sample_rows(torch.zeros(rows, 151936), torch.zeros(7, rows, dtype=torch.int32))
    assert asked[0][8] == first | second << 1
    assert kernels.launch_count() - before == launches
