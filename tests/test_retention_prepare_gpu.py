"""Preparing q and k of retention: rows on boundaries of four values go to a kernel of their own, which has to give the general
one's bits."""

import ctypes

import pytest
import torch

from tinyvllm_b200.ops import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,dim,rot,pairing", [(1, 1, 4, None, 0), (3, 2, 8, 8, 1), (5, 3, 12, 8, 1), (5, 3, 12, 4, 0),
                                                          (7, 2, 20, 12, 0), (1030, 4, 128, 128, 1), (9, 16, 128, 64, 1),
                                                          (33, 3, 36, 36, 0), (2, 1, 256, 256, 0)])
def test_both_forms_give_the_same_bits(dtype, tokens, heads, dim, rot, pairing):
    from ctypes import c_float, c_int, c_longlong, c_void_p

    g = torch.Generator(device=DEV).manual_seed(dim + tokens)
    per, tag = heads * dim, 0 if dtype == torch.float32 else 1
    fn = kernels._fn("retention", "tvb_retention_prepare",
                     [c_void_p, c_longlong] + [c_int] * 4 + [c_void_p, c_int, c_int, c_float] + [c_void_p] * 3
                     + [c_int, c_int, c_void_p])
    inv_freq = None if rot is None else 10000.0 ** (-2.0 * torch.arange(rot // 2, device=DEV) / rot)
    positions = torch.randint(0, 5000, (tokens,), generator=g, device=DEV, dtype=torch.int32)
    values = torch.randn(tokens, 2 * per, generator=g, device=DEV).to(dtype)
    got = []
    for shift in (0, 1):                                       # off the boundary: the general kernel
        stride = 2 * per + 8
        proj = torch.zeros(tokens, stride, dtype=dtype, device=DEV)
        proj[:, 4 + shift:4 + shift + 2 * per] = values
        q, k = (torch.full((tokens, per), float("nan"), device=DEV) for _ in range(2))
        assert fn(proj.data_ptr(), stride, 4 + shift, 4 + shift + per, heads, dim,
                  None if inv_freq is None else inv_freq.data_ptr(), rot or 0, pairing, 0.25, positions.data_ptr(),
                  q.data_ptr(), k.data_ptr(), tokens, tag, torch.cuda.current_stream().cuda_stream) == 0
        got.append((q, k))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and not got[0][0].isnan().any()
