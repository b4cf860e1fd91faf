"""The scratch of float32 products is bounded, whatever their sizes.  No GPU."""

import pytest

from tinyvllm_b200.ops import kernels

WEIGHTS = [(4096, 1024), (1024, 2048), (6144, 1024), (1024, 3072), (151936, 1024), (24576, 4096), (4096, 12288), (51200, 5120),
           (5120, 25600), (151936, 5120), (64, 1 << 20), (7, 513), (1 << 20, 513)]


@pytest.mark.parametrize("n,k", WEIGHTS)
def test_partial_sums_take_at_most_64_mib(n, k):
    for m in (1, 8, 9, 16, 17, 33, 48, 64, 65, 130, 300, 512, 677, 1024, 2048, 4096, 8192, 16384, 1 << 20):
        assert 0 <= 4 * kernels.gemm_f32_scratch_floats(m, n, k) <= 64 << 20, m


def test_products_that_leave_the_gpu_idle_are_cut():
    """... and those that fill it are not."""
    assert kernels.gemm_f32_scratch_floats(300, 1024, 2048) == 4 * 300 * 1024
    assert kernels.gemm_f32_scratch_floats(2048, 6144, 1024) == 0
