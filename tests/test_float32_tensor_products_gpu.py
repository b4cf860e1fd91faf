"""Products of float32 operands on the tensor cores: against 64 bits at the edges of tiles, blocks and groups of k, values
that have no three bfloat16 parts, products at the end of the float32 range, and that a row's sum does not depend on the other
rows."""

import pytest
import torch

from tinyvllm_b200.ops import kernels, linear

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def bound(a, w):
    """A block of 64 k: 4 products that the tensor cores cut at 2^-23 of the sum so far (twice, for the small ones before
    them), then one rounding a block and a group; the parts left out, x2 w3 and x3 w2, are 2^-8 2^-16 of a product each at
    most, together 2 units of 2^-24."""
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


def draw_operands(kind, n, k, generator):
    def normal(rows):
        return torch.randn(rows, k, generator=generator, device=DEV)

    def uniform(rows):
        return torch.rand(rows, k, generator=generator, device=DEV)

    if kind == "normal":
        return normal(n), normal(n) * 0.02
    if kind == "long tails":
        return normal(n) * torch.exp(2 * normal(n)), normal(n) * 0.02
    if kind == "one sign by either":
        return uniform(n), normal(n)
    if kind == "one sign":
        return uniform(n), uniform(n)
    if kind == "one sign, long tails":
        return torch.exp(2 * normal(n)), torch.exp(2 * normal(n))
    if kind == "rows of one value":
        return (uniform(n)[:, :1] + 0.5).expand(n, k).contiguous(), (uniform(n)[:, :1] + 0.5).expand(n, k).contiguous()
    # every part left out has the sign and nearly the size of the largest there is
    return (torch.full((n, k), 1.0 + 2.0 ** -8 - 2.0 ** -23, device=DEV),) * 2


@pytest.mark.parametrize("k", [4, 12, 16, 64, 128, 1024, 2052])
@pytest.mark.parametrize("kind", ["normal", "long tails", "one sign by either", "one sign", "one sign, long tails", "rows of one value",
                                  "largest left out"])
def test_error_against_64_bits_beside_the_float32_cores(kind, k):
    generator = torch.Generator(device=DEV).manual_seed(k)
    a, w = draw_operands(kind, 256, k, generator)
    want = a.double() @ w.double().T
    errors = []
    for product in (kernels.gemm_f32_tc, kernels.gemm_nt_simt):
        off = product(a, w).double() - want
        assert product is kernels.gemm_nt_simt or (off.abs() <= bound(a, w)).all()
        errors.append((off.norm() / want.norm()).item())
    # weights of either sign, as a model's: no further off than the float32 cores from the k on that the tensor cores take
    # (measured 0.44 to 0.98 of it; long tails at 64 k hang on few products: 1.07)
    if kind in ("normal", "one sign by either") and k >= 16 or kind in ("long tails", "rows of one value") and k >= 128:
        assert errors[0] <= errors[1], errors


def test_sums_that_fit_24_bits_are_exact():
    generator = torch.Generator(device=DEV).manual_seed(8)
    a, w = (torch.randint(-50, 51, (130, 3072), generator=generator, device=DEV).float() for _ in range(2))
    assert torch.equal(kernels.gemm_f32_tc(a, w).double(), a.double() @ w.double().T)
    x = torch.randn(70, 256, generator=generator, device=DEV) * 1e-20
    assert torch.equal(kernels.gemm_f32_tc(x, torch.eye(256, device=DEV)), x)


def test_rounding_changes_where_the_kernel_does():
    """32 rows are the float32 cores', 33 the tensor cores': a row differs by no more than both kernels' errors."""
    generator = torch.Generator(device=DEV).manual_seed(9)
    a, w = torch.randn(33, 1024, generator=generator, device=DEV), torch.randn(1024, 1024, generator=generator, device=DEV)
    few, more = linear(a[:32], w), linear(a, w)[:32]
    assert torch.equal(few, kernels.gemm_nt_simt(a[:32], w)) and torch.equal(more, kernels.gemm_f32_tc(a, w)[:32])
    # a chain of 64 products, the sum of two chains, 3 segments and 2 groups on the float32 cores
    cores = (64 + 1 + 3 + 2) * 2.0 ** -24 * (a[:32].double().abs() @ w.double().abs().T)
    assert ((few.double() - more.double()).abs() <= cores + bound(a[:32], w)).all()


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


def same_where_not_finite(got, want):
    return torch.equal(got.isnan(), want.isnan()) and torch.equal(got == float("inf"), want == float("inf")) and torch.equal(
        got == float("-inf"), want == float("-inf"))


@pytest.mark.parametrize("m,n,k", [(40, 130, 64), (150, 140, 1028), (150, 140, 2048), (2500, 1500, 2052), (1100, 40, 25600)])
def test_products_beyond_float32_are_summed_as_the_float32_cores_do(m, n, k):
    """Finite operands whose products, or parts' products, leave float32: whole, cut and added up from partial sums, in ranges of rows."""
    generator = torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(m, k, generator=generator, device=DEV), torch.randn(n, k, generator=generator, device=DEV)
    a, w = a + a.sign(), w + w.sign()                       # none near zero: every product below is beyond float32
    for scale in (1e20, 1e21, 3e37):
        got, want = kernels.gemm_f32_tc(a * scale, w * scale), kernels.gemm_nt_simt(a * scale, w * scale)
        assert same_where_not_finite(got, want) and not want.isfinite().any(), scale
    # a row and a column of them, the rest as ever
    clean, some = kernels.gemm_f32_tc(a, w), a.clone()
    some[m - 3] *= 1e38
    got, want = kernels.gemm_f32_tc(some, w), kernels.gemm_nt_simt(some, w)
    kept = torch.arange(m, device=DEV) != m - 3
    assert torch.equal(got[kept], clean[kept]) and same_where_not_finite(got, want)
    # a NaN in a row, infinities of either sign in another and in a column
    some = a.clone()
    some[3, 7], some[20, k - 1], some[20, 0] = float("nan"), float("inf"), float("-inf")
    wide = w.clone()
    wide[11, 5] = float("inf")
    got, want = kernels.gemm_f32_tc(some, wide), kernels.gemm_nt_simt(some, wide)
    assert same_where_not_finite(got, want) and got[3].isnan().all()
    kept[m - 3], kept[3], kept[20] = True, False, False
    others = torch.arange(n, device=DEV) != 11
    assert torch.equal(got[kept][:, others], clean[kept][:, others])


@pytest.mark.parametrize("k", [64, 1024, 2048])
def test_products_just_inside_float32(k):
    """u * v up to the largest float32: the first parts round up and their product is beyond it.  Alone, and two that cancel."""
    generator = torch.Generator(device=DEV).manual_seed(k + 1)
    largest = torch.finfo(torch.float32).max
    u = (1.0 + torch.rand(150, generator=generator, device=DEV, dtype=torch.float64)).float()
    v = (1.06 - 0.08 * torch.rand(140, generator=generator, device=DEV, dtype=torch.float64)).float()
    u[:75] = 2.0 - 0.008 * (u[:75] - 1.0)
    a, w = torch.zeros(150, k, device=DEV), torch.zeros(140, k, device=DEV)
    a[:, 5], w[:, 5] = u * 2.0 ** 63, v * 2.0 ** 64          # products from 2^126 to beyond the largest float32, many near it
    want = a[:, 5:6].double() @ w[:, 5:6].double().T
    inside = want.abs() <= largest
    near = inside & (want.abs() > 0.98 * largest)
    assert near.sum() > 100 and not inside.all()
    got = kernels.gemm_f32_tc(a, w)
    assert got[inside].isfinite().all() and got[~inside & (want > 1.0001 * largest)].isinf().all()
    assert ((got.double() - want).abs()[inside] <= bound(a, w)[inside]).all()
    a[:, k - 2], w[:, k - 2] = a[:, 5], -w[:, 5]             # the same once more with the other sign, far along k
    got = kernels.gemm_f32_tc(a, w)
    assert (got[inside].abs() <= bound(a, w)[inside]).all() and torch.equal(got[near], kernels.gemm_nt_simt(a, w)[near])


@pytest.mark.parametrize("m,k", [(64, 512), (301, 2052)])
@pytest.mark.parametrize("scale", [1e-42, 1e-40, 1e-38, 1e-36, 1e-34, 1e-30, 1e-18, 1e18, 1e26, 1e30, 1e36])
@pytest.mark.parametrize("of_a", [True, False])
def test_large_and_small_values(m, k, scale, of_a):
    generator = torch.Generator(device=DEV).manual_seed(3)
    a, w = torch.randn(m, k, generator=generator, device=DEV), torch.randn(96, k, generator=generator, device=DEV)
    if of_a:
        a *= scale
    else:
        w *= scale
    want = a.double() @ w.double().T
    got = kernels.gemm_f32_tc(a, w)
    # below 2^-126 a sum of a group and theirs round to multiples of 2^-149
    assert ((got.double() - want).abs() <= bound(a, w) + 2 * -(-k // 1024) * 2.0 ** -150).all()
    if scale >= 1e36:                                       # sums beyond 2^96 are the float32 cores'
        huge = want.abs() > 2.0 ** 97
        assert huge.float().mean() > 0.9 and torch.equal(got[huge], kernels.gemm_nt_simt(a, w)[huge])


@pytest.mark.parametrize("scales", [(1e-20, 1e-20), (1e-25, 1e-15), (1e-30, 1e-12), (1e-42, 1e3), (1e14, 1e14)])
def test_products_at_the_ends_of_float32(scales):
    """Both operands small, or both large: sums down to the smallest float32 and beyond 2^96."""
    generator = torch.Generator(device=DEV).manual_seed(4)
    a = torch.randn(64, 512, generator=generator, device=DEV) * scales[0]
    w = torch.randn(96, 512, generator=generator, device=DEV) * scales[1]
    want = a.double() @ w.double().T
    for got in (kernels.gemm_f32_tc(a, w), kernels.gemm_f32_tc(a.repeat(3, 1), w)[128:]):
        # (a product of two parts below 2^-149 / 2^32 is nothing to a multiple of 2^-149)
        assert ((got.double() - want).abs() <= bound(a, w) + 2.0 ** -149).all()


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
