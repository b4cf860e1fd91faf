"""Which float32 products may read their weight before the kernel before them has ended: those of the parts, whose weights are
parameters, and no other.  No GPU."""

import ast
from pathlib import Path

import pytest
import torch

from tinyvllm_b200.ops import kernels
from tinyvllm_b200.ops import linear as exported
from tinyvllm_b200.ops.linear import linear, linear_into_stream, linear_norm, linear_silu

PACKAGE = Path(kernels.__file__).resolve().parent.parent
FUNCTIONS = ("linear", "linear_silu", "linear_norm", "linear_into_stream")


class OnGpu(torch.Tensor):
    is_cuda = True


class Norm:
    def forward(self, x):
        return x

    def add(self, x, residual):
        return x, residual


@pytest.mark.parametrize("rows", [1, 8, 32, 33, 200])
@pytest.mark.parametrize("given", [{}, {"weight_constant": False}, {"weight_constant": True}])
def test_the_caller_says_it(monkeypatch, rows, given):
    seen = []

    def product(a, w, out=None, weight_constant=False):
        seen.append(weight_constant)
        return torch.zeros(a.shape[0], w.shape[0])

    monkeypatch.setattr(kernels, "gemm_nt_simt", product)
    monkeypatch.setattr(kernels, "gemm_f32_tc", product)
    monkeypatch.setattr(kernels, "silu_mul", lambda packed: packed)
    x, w = torch.zeros(rows, 64).as_subclass(OnGpu), torch.zeros(48, 64)
    linear(x, w, **given)
    linear_silu(x, w, **given)
    linear_into_stream(x, w, None, **given)
    for silu in (False, True):
        linear_norm(x, None, Norm(), w, silu=silu, **given)
        linear_norm(None, x, Norm(), w, silu=silu, **given)
    assert seen == [given.get("weight_constant", False)] * 7
    assert exported is linear


def test_the_parts_say_that_their_weights_are():
    calls = 0
    for path in [*sorted((PACKAGE / "parts").glob("*.py")), PACKAGE / "ops" / "attention.py"]:
        for node in ast.walk(ast.parse(path.read_text())):
            if isinstance(node, ast.Call) and isinstance(node.func, ast.Name) and node.func.id in FUNCTIONS:
                calls += 1
                assert any(word.arg == "weight_constant" for word in node.keywords), (path.name, node.lineno)
    assert calls > 30
