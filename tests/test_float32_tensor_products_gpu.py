"""Products of float32 operands on the tensor cores: against 64 bits at the edges of tiles, blocks and groups of k, values
that have no three bfloat16 parts, and that a row's sum does not depend on the other rows."""

import pytest
import torch

from tinyvllm_b200.ops import kernels, linear

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bound(a, w):
    """A block of 64 k: 4 products that the tensor cores cut at 2^-23 of the sum so far (twice, for the small ones before
    them), then one rounding a block and a group; the parts left out are 2^-24 of a product at most."""
    k = a.shape[1]
    return (8 * 2.0 ** -23 + (-(-min(k, 1024) // 64) + -(-k // 1024) + 2) * 2.0 ** -24) * (a.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("n,k", [(1, 4), (7, 60), (128, 64), (129, 68), (130, 1028), (1024, 3072), (520, 1024), (257, 2052)])
def test_sums_are_within_float32_and_the_same_in_every_batch(n, k):
    generator = torch.Generator(device=DEV).manual_seed(n + k)
    a = torch.randn(331, k, generator=generator, device=DEV)
    w = torch.randn(n, k, generator=generator, device=DEV)
    whole = kernels.gemm_f32_tc(a, w)
    want = a.double() @ w.double().T
    assert ((whole.double() - want).abs() <= bound(a, w)).all()
    for rows in (1, 15, 16, 17, 33, 64, 127, 128, 129, 200):
        assert torch.equal(kernels.gemm_f32_tc(a[:rows], w), whole[:rows]), rows
    # rows apart, and a result inside a wider tensor
    apart = torch.empty(331, k + 8, device=DEV)[:, 4:k + 4].copy_(a)
    into = torch.full((331, n + 5), 7.0, device=DEV)
    kernels.gemm_f32_tc(apart, w, out=into[:, 2:n + 2])
    assert torch.equal(into[:, 2:n + 2], whole) and (into[:, :2] == 7.0).all() and (into[:, n + 2:] == 7.0).all()
    assert kernels.gemm_f32_tc_status() == 0


@pytest.mark.parametrize("k", [64, 2048])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38, -3.395e38])
def test_values_without_three_parts(value, k):
    generator = torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(150, k, generator=generator, device=DEV), torch.randn(140, k, generator=generator, device=DEV)
    w[w.abs() < 0.5] = 0.5                                  # (no sum of huge values comes near zero)
    clean = kernels.gemm_f32_tc(a, w)
    wild_a, wild_w = a.clone(), w.clone()
    wild_a[137, k - 3], wild_w[70, 5] = value, value
    if abs(value) < float("inf"):
        wild_w[70, 5] = value * 1e-3
        wild_a[:, 5] *= 1e-3
    got, want = kernels.gemm_f32_tc(wild_a, wild_w), (wild_a.double() @ wild_w.double().T).float()
    rows, cols = torch.arange(150, device=DEV) != 137, torch.arange(140, device=DEV) != 70
    if abs(value) == float("inf") or value != value:
        assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    for at in (got[137] - want[137], got[:, 70] - want[:, 70]):
        same = torch.isfinite(at)
        assert (at[same].abs() <= 1e-5 * k * max(1.0, 1e36 if abs(value) < float("inf") else 1.0)).all()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())


@pytest.mark.parametrize("scale", [1e-30, 1e-18, 1e18, 1e30])
def test_large_and_small_values(scale):
    generator = torch.Generator(device=DEV).manual_seed(3)
    a, w = torch.randn(64, 512, generator=generator, device=DEV) * scale, torch.randn(96, 512, generator=generator, device=DEV)
    want = a.double() @ w.double().T
    got = kernels.gemm_f32_tc(a, w).double()
    assert ((got - want).abs() <= bound(a, w)).all()


def test_which_kernel_takes_a_product():
    generator = torch.Generator(device=DEV).manual_seed(5)
    a, w = torch.randn(80, 128, generator=generator, device=DEV), torch.randn(72, 128, generator=generator, device=DEV)
    assert torch.equal(linear(a, w), kernels.gemm_f32_tc(a, w))
    assert torch.equal(linear(a[:32], w), kernels.gemm_nt_simt(a[:32], w))
    off = torch.randn(80 * 128 + 1, generator=generator, device=DEV)[1:].view(80, 128)          # off the 16-byte boundary
    assert torch.equal(linear(off, w), kernels.gemm_nt_simt(off, w))
    odd = a[:, :127].contiguous()
    assert torch.equal(linear(odd, w[:, :127].contiguous()), kernels.gemm_nt_simt(odd, w[:, :127].contiguous()))


def test_products_in_ranges_of_rows():
    """More rows than 64 MiB of parts hold: the ranges' sums are those of a product of their own."""
    generator = torch.Generator(device=DEV).manual_seed(6)
    a = torch.randn(1100, 25600, generator=generator, device=DEV)
    w = torch.randn(40, 25600, generator=generator, device=DEV)
    whole = kernels.gemm_f32_tc(a, w)
    assert torch.equal(whole[1000:], kernels.gemm_f32_tc(a[1000:], w)) and torch.equal(whole[:50], kernels.gemm_f32_tc(a[:50], w))
    assert ((whole.double() - a.double() @ w.double().T).abs() <= bound(a, w)).all()
