"""The RMS norm on weights that the launch just before it writes: it may start while that one still runs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [64, 1024, 4096])
def test_weights_of_the_launch_before_are_awaited(width):
    from tinyvllm_b200.ops import kernels

    generator = torch.Generator().manual_seed(width)
    x = torch.randn(3000, width, generator=generator).bfloat16().cuda()
    rows = torch.randn(5, width, generator=generator).bfloat16().cuda()
    ones = torch.ones(width, device="cuda")
    made = torch.empty_like(x)
    for turn in range(40):
        made.fill_(50.0)                            # what a reader ahead of the store would see
        weights = torch.randn(width, generator=generator).cuda()
        kernels.rms_norm(x, weights, 1e-6, out=made)
        got = kernels.rms_norm(rows, made[2999 - turn], 1e-6)
        assert torch.equal(got, kernels.rms_norm(rows, made[2999 - turn].clone(), 1e-6)), turn
        want = rows.float() * torch.rsqrt(rows.float().square().mean(1, keepdim=True) + 1e-6)
        want = want.bfloat16().float() * made[2999 - turn].float()
        # two roundings to bfloat16, the first of a value that may fall on either side (one step of 2^-7)
        assert ((got.float() - want).abs() <= want.abs() * 2.0 ** -6 + 1e-6).all(), turn
    assert kernels.rms_norm(rows, ones, 1e-6).isfinite().all()
