"""Products of float32 operands: every form of the kernels (few rows, tiles, cut sums, rows off the 16-byte boundary)
against 64 bits, and that a row's sum has the same bits in all of them."""

import pytest
import torch

from tinyvllm_b200.ops import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,k", [(1, 1), (7, 127), (65, 128), (130, 516), (1024, 3072), (520, 1024), (4736, 260), (5003, 2044),
                                 (24, 25600), (5003, 5632)])
def test_every_form_gives_a_row_the_same_bits(n, k):
    generator = torch.Generator(device=DEV).manual_seed(n + k)
    a = torch.randn(331, k, generator=generator, device=DEV)
    w = torch.randn(n, k, generator=generator, device=DEV)
    whole = kernels.gemm_nt_simt(a, w)
    want = a.double() @ w.double().T
    # at most 64 products in a chain, the two chains' sum, 3 segments and the groups: each adds half a unit of the absolute sum
    bound = (64 + 1 + 3 + -(-k // 512)) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert ((whole.double() - want).abs() <= bound).all()
    for rows in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 130):
        assert torch.equal(kernels.gemm_nt_simt(a[:rows], w), whole[:rows]), rows
    # rows that start off the 16-byte boundary, and a result inside a wider tensor
    shifted = torch.empty(331, k + 3, device=DEV)[:, 1:k + 1].copy_(a)
    into = torch.full((331, n + 5), 7.0, device=DEV)
    for rows in (3, 331):
        kernels.gemm_nt_simt(shifted[:rows], w, out=into[:rows, 2:n + 2])
        assert torch.equal(into[:rows, 2:n + 2], whole[:rows])
    assert (into[:, :2] == 7.0).all() and (into[:, n + 2:] == 7.0).all()
    # a row outside the product, whatever it holds, touches no other
    wild = a.clone()
    wild[5] = float("nan")
    got = kernels.gemm_nt_simt(wild[:7], w)
    assert torch.equal(got[[0, 1, 2, 3, 4, 6]], whole[[0, 1, 2, 3, 4, 6]]) and got[5].isnan().all()
