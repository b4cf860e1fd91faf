"""The scratch of float32 products on the tensor cores is bounded, whatever their sizes.  No GPU."""

import pytest

from tinyvllm_b200.ops import kernels
from test_float32_scratch import WEIGHTS


@pytest.mark.parametrize("n,k", WEIGHTS)
def test_partial_sums_and_parts_take_at_most_64_mib_each(n, k):
    parts_of_128 = 128 * (6 * (-(-k // 64) * 64) + 4)
    for m in (1, 33, 128, 129, 677, 2048, 8192, 16384, 16385, 1 << 20):
        assert 0 < kernels.gemm_f32_tc_scratch_bytes(m, n, k) <= (64 << 20) + max((64 << 20) + (1 << 20), parts_of_128), m
