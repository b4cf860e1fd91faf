"""The decode attention on tokens whose keys the launch just before it stores: the rest of a short
prompt portion is normalised, rotated and stored by one kernel and attended by the next, which may
start while the first still runs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 2, 3])
def test_keys_of_the_launch_before_are_awaited(tokens):
    from tinyvllm_b200.ops import kernels

    dim, num_q, num_kv, page = 128, 8, 2, 32
    generator = torch.Generator().manual_seed(tokens)
    cos, sin = torch.ones(64, dim // 2, device="cuda"), torch.zeros(64, dim // 2, device="cuda")
    weight = torch.ones(dim, device="cuda")
    positions = torch.arange(tokens, dtype=torch.int32, device="cuda")
    rows = torch.zeros(tokens, dtype=torch.int32, device="cuda")
    table = torch.zeros((1, 8), dtype=torch.int32, device="cuda")
    caches = [torch.zeros((1, num_kv, page, dim), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    heads = dict(num_q=num_q, num_kv=num_kv, head_dim=dim)
    for _ in range(40):
        qkv = torch.randn((tokens, (num_q + 2 * num_kv) * dim), generator=generator).to(torch.bfloat16).cuda()
        for cache in caches:
            cache.fill_(50.0)                       # what a reader ahead of the store would see
        kernels.qk_norm_rope_store(qkv, **heads, positions=positions, q_weight=weight, k_weight=weight, eps=1e-6, cos=cos,
                                   sin=sin, slots=positions, key_cache=caches[0], value_cache=caches[1])
        got = kernels.attention_decode(qkv, **heads, positions=positions, token_row=rows, slots=None, q_weight=None,
                                       k_weight=None, eps=0.0, cos=None, sin=None, key_cache=caches[0],
                                       value_cache=caches[1], block_tables=table, window=None, scale=dim ** -0.5,
                                       splits=4, max_context=64, new_in_cache=True, library_of=torch.float32)
        q = qkv[:, :num_q * dim].float().view(tokens, num_q, dim)
        k, v = (cache[0, :, :tokens].float().repeat_interleave(num_q // num_kv, 0) for cache in caches)
        scores = torch.einsum("ihd,hjd->hij", q, k) * dim ** -0.5
        scores = scores.masked_fill(torch.ones(tokens, tokens, device="cuda").triu(1).bool(), -torch.inf)
        want = torch.einsum("hij,hjd->ihd", torch.softmax(scores, -1), v).reshape(tokens, -1)
        # weights and result are rounded to bfloat16 once each (2^-9 of values below about 4), stale keys are 50 off
        assert (got.float() - want).abs().max().item() <= 0.05
