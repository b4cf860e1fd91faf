"""The RMS norm of float32 rows: the register form at the edges of its widths, the general one beside it, and weights that
the launch before writes (of the norm and of products of a few rows)."""

import pytest
import torch

from tinyvllm_b200.ops import kernels, linear, linear_into_stream, linear_silu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [4, 31, 36, 1020, 1024, 1028, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("constant", [False, True])
def test_against_64_bits(width, constant):
    generator = torch.Generator(device="cuda").manual_seed(width)
    x, r = (torch.randn(37, width, generator=generator, device="cuda") for _ in range(2))
    weight = torch.randn(width, generator=generator, device="cuda")
    got, stream = kernels.rms_norm(x, weight, 1e-6, residual=r, weight_constant=constant)
    assert torch.equal(stream, x + r)
    wide = (x + r).double()
    want = wide / (wide.square().mean(1, keepdim=True) + 1e-6).sqrt() * weight.double()
    # the sum of squares over chains of at most 16 and 9 halvings, its root, the quotient and two products
    assert ((got.double() - want).abs() <= 32 * 2.0 ** -24 * want.abs()).all()
    rows = torch.tensor([36, 0, 5], dtype=torch.int32, device="cuda")
    assert torch.equal(kernels.rms_norm(x + r, weight, 1e-6, rows=rows), got[rows.long()])
    shifted = torch.empty(37 * width + 1, device="cuda")[1:].view(37, width).copy_(x + r)          # off the 16-byte boundary
    assert ((kernels.rms_norm(shifted, weight, 1e-6).double() - want).abs() <= 32 * 2.0 ** -24 * want.abs()).all()


@pytest.mark.parametrize("width", [64, 1024, 4096])
def test_weights_and_products_of_the_launch_before_are_awaited(width):
    generator = torch.Generator(device="cuda").manual_seed(width)
    x = torch.randn(3000, width, generator=generator, device="cuda")
    rows = torch.randn(5, width, generator=generator, device="cuda")
    made = torch.empty_like(x)
    for turn in range(40):
        made.fill_(50.0)                            # what a reader ahead of the store would see
        weight = torch.randn(width, generator=generator, device="cuda")
        kernels.rms_norm(x, weight, 1e-6, out=made)
        got = kernels.rms_norm(rows, made[2999 - turn], 1e-6)
        assert torch.equal(got, kernels.rms_norm(rows, made[2999 - turn].clone(), 1e-6)), turn
        made.fill_(50.0)
        kernels.rms_norm(x, weight, 1e-6, out=made)
        got = kernels.gemm_nt_simt(rows, made[2900:])                # a weight that the launch before writes
        assert torch.equal(got, kernels.gemm_nt_simt(rows, made[2900:].clone())), turn


@pytest.mark.parametrize("rows", [1, 5, 8, 20, 64, 200])
def test_linear_awaits_a_weight_that_the_launch_before_writes(rows):
    """Without weight_constant a weight may come from the launch before, whatever kernel takes the product."""
    generator = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(6000, 1024, generator=generator, device="cuda")
    few = torch.randn(rows, 1024, generator=generator, device="cuda")
    made = torch.empty_like(x)
    for turn in range(30):
        made.fill_(50.0)
        norm = torch.randn(1024, generator=generator, device="cuda")
        kernels.rms_norm(x, norm, 1e-6, out=made)              # (lets what is launched behind it begin early)
        got = linear(few, made[5000:])
        assert torch.equal(got, linear(few, made[5000:].clone())), turn
    made.fill_(50.0)
    kernels.rms_norm(x, norm, 1e-6, out=made)
    got = linear_silu(few, made[5000:])
    assert torch.equal(got, linear_silu(few, made[5000:].clone()))
    made.fill_(50.0)
    kernels.rms_norm(x, norm, 1e-6, out=made)
    got = linear_into_stream(few, made[4976:], few)[0]
    assert torch.equal(got, linear_into_stream(few, made[4976:].clone(), few)[0])


@pytest.mark.parametrize("inter", [1, 6, 8, 1020, 1028, 3072])
def test_silu_times_up(inter):
    generator = torch.Generator(device="cuda").manual_seed(inter)
    packed = torch.randn(5, 2 * inter, generator=generator, device="cuda") * 4
    gate, up = packed.double().split(inter, dim=1)
    want = gate / (1 + torch.exp(-gate)) * up
    for rows in (packed, torch.empty(10 * inter + 1, device="cuda")[1:].view(5, 2 * inter).copy_(packed)):   # (off the boundary)
        assert ((kernels.silu_mul(rows).double() - want).abs() <= 8 * 2.0 ** -24 * want.abs() + 1e-37).all()
