"""The tcgen05 prefill attention with windows that keep first keys, segments, sinks, a learned bias by distance and gates,
against 64-bit sums, over pages whose unused slots hold NaN."""

import pytest
import torch

from test_kernels_gpu import DEV, k

pytestmark = pytest.mark.gpu

FORMS = {
    "window": dict(window=70), "window-kept": dict(window=300, keep=4), "kept-blocks": dict(window=40, keep=200),
    "one-key": dict(window=1, keep=1), "full": dict(), "segments": dict(segment=192), "long-segments": dict(segment=1024),
    "bias": dict(bias=33), "bias-sink-segments": dict(bias=257, sink=True, segment=256, gate="value"),
    "sink": dict(sink=True, window=130, keep=3), "gates": dict(gate="value", window=130), "head-gates": dict(gate="head"),
    "long-bias": dict(bias=2048, sink=True, gate="value", odd=True),
}


@pytest.mark.parametrize("shape", [(1, 1, 16), (4, 2, 16), (16, 8, 8), (6, 2, 128)])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_against_64_bits(form, shape):
    from tinyvllm_b200.ops.attention import prefill_tiles

    nq, nkv, page = shape
    window, keep, segment, bias, sink, gate, odd = (FORMS[form].get(name) for name in (
        "window", "keep", "segment", "bias", "sink", "gate", "odd"))
    g = torch.Generator().manual_seed(len(form) + nq)
    lengths, counts = [700, 131, 96, 1300], [513, 131, 40, 160]
    pages = sum(-(-n // page) for n in lengths) + 2
    order = torch.randperm(pages, generator=g).tolist()
    if page == 16:
        order = sorted(order, reverse=True)                # pages one behind the other: copied in pairs
    kc = torch.full((pages, nkv, page, 128), float("nan"), dtype=torch.bfloat16)
    vc = kc.clone()
    tables = torch.full((4, max(-(-n // page) for n in lengths)), -1, dtype=torch.int32)
    q_rows, token_row, positions, keys, values = [], [], [], [], []
    for r, (n, count) in enumerate(zip(lengths, counts)):
        kr, vr = (torch.randn(n, nkv, 128, generator=g).bfloat16() for _ in range(2))
        keys.append(kr.double()), values.append(vr.double())
        for b in range(-(-n // page)):
            tables[r, b] = order.pop()
            span = slice(b * page, min(n, (b + 1) * page))
            kc[tables[r, b], :, :span.stop - span.start] = kr[span].transpose(0, 1)
            vc[tables[r, b], :, :span.stop - span.start] = vr[span].transpose(0, 1)
        q_rows.append(torch.randn(count, nq, 128, generator=g).bfloat16())
        token_row += [r] * count
        positions += list(range(n - count, n))
    q = torch.cat(q_rows)
    tokens, scale = q.shape[0], 0.11
    table = torch.randn(bias, nq, generator=g) if bias else None
    sinks = torch.randn(nq, generator=g) * 3 if sink else None
    gates = torch.randn(tokens, (nq if gate == "head" else nq * 128) + (3 if odd else 0), generator=g).bfloat16() if gate else None
    if odd and gate:
        gates = gates[:, 3:]
    big, rest, _ = prefill_tiles(counts, [n - c for n, c in zip(lengths, counts)], tensor_memory=True)
    out = torch.full((tokens, nq * 128 + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    where = lambda t: None if t is None else t.to(DEV)
    gate_in = None
    if gates is not None:                                  # on the device with the offset that it has here
        gate_in = torch.empty(tokens, gates.stride(0), dtype=torch.bfloat16, device=DEV)[:, gates.stride(0) - gates.shape[1]:]
        gate_in.copy_(gates)
    k().attention_prefill_tc_extras(
        q.view(tokens, -1).to(DEV), kc.to(DEV), vc.to(DEV), tables.to(DEV), i32(positions), *map(i32, big), num_q=nq,
        num_kv=nkv, key_dim=128, value_dim=128, window=window, keep_first=keep or 0, scale=scale, out=out[:, :nq * 128],
        gate=gate_in, gate_per_head=gate == "head", sinks=where(sinks), bias_table=where(table), segment=segment)
    assert k().attention_prefill_tc_status() == 0
    got = out.cpu()[:, :nq * 128].double().view(tokens, nq, 128)
    assert out[:, nq * 128:].isnan().all()
    tiled = torch.zeros(tokens, dtype=torch.bool)
    for first, count in zip(big[1], big[2]):
        tiled[first:first + count] = True
    at = 0
    for r, (n, count) in enumerate(zip(lengths, counts)):
        i = torch.arange(n - count, n)[:, None]
        j = torch.arange(n)[None, :]
        seen = j <= i
        if segment:
            seen &= j >= i - i % segment
        if window:
            seen &= (i - j < window) | (j < (keep or 0))
        for h in range(nq):
            s = (q[at:at + count, h].double() @ keys[r][:, h // (nq // nkv)].T) * scale
            if table is not None:
                s = s + table[(i - j).clamp(0, bias - 1), h].double()
            s = s.masked_fill(~seen, -torch.inf)
            top = s.amax(1, keepdim=True)
            e = torch.exp(s - top)
            total = e.sum(1, keepdim=True)
            if sinks is not None:
                total = total + torch.exp(sinks[h].double() - top)
            p = e / total
            want, size = p @ values[r][:, h // (nq // nkv)], p @ values[r][:, h // (nq // nkv)].abs()
            if gate:
                lift = torch.sigmoid(gates[at:at + count, [h]].double() if gate == "head" else
                                     gates[at:at + count, h * 128:(h + 1) * 128].double())
                want, size = want * lift, size * lift
            mine = tiled[at:at + count]
            # the result's rounding to 16 bits, the weights' 2^-17 and float32 scores up to about 30
            bound = want.abs() * 2.0 ** -8 + size * 2.0 ** -15
            assert ((got[at:at + count, h] - want).abs() <= bound)[mine].all(), (r, h)
        at += count
    assert got[~tiled].isnan().all()                       # tokens of no tile are left alone
