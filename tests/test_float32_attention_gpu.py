"""Float32 attention over whole heads of 64 and 128: the kernel for tiles of tokens, the kernel for single tokens and their
mixes against the plain implementation, and that a token's result has the same bits however the tokens come."""

import pytest
import torch

from test_kernels_gpu import DEV, close, k, paged_case, plain_paged, run_rows

pytestmark = pytest.mark.gpu


def some_rows(case, rows):
    picked = dict(case)
    for name in ("q", "token_row", "positions"):
        picked[name] = case[name][rows].contiguous()
    return picked


@pytest.mark.parametrize("window", [None, 100, 300])
@pytest.mark.parametrize("heads", [(2, 2, 128), (4, 2, 128), (8, 2, 64), (8, 1, 128), (3, 3, 64), (4, 2, 64), (4, 1, 128), (8, 1, 64)])
def test_tiles_and_single_tokens_agree(heads, window):
    nq, nkv, d = heads
    case = paged_case(torch.float32, nq=nq, nkv=nkv, d=d, page=16, lengths=[300, 1, 70, 515, 257, 640, 33],
                      queries=[40, 1, 3, 5, 257, 129, 33], seed=nq + d)
    shape = dict(nq=nq, nkv=nkv, d=d, scale=d ** -0.5, window=window)
    want = plain_paged(case, d ** -0.5, window, torch.float32)
    walked = run_rows(case, **shape, max_chunks=0)
    close(walked, want, torch.float32, f32=3e-6, bf16=0)
    assert torch.equal(run_rows(case, **shape, max_chunks=3), walked)
    total = walked.shape[0]
    for rows in (slice(0, 1), slice(39, 45), slice(41, 50), slice(48, 49), slice(30, 62), slice(total - 40, total),
                 slice(0, total, 3)):
        part = some_rows(case, rows)
        for chunks in (0, 3):
            assert torch.equal(run_rows(part, **shape, max_chunks=chunks), walked[rows]), (rows, chunks)
    # padding rows are zero and change no other
    padded = some_rows(case, slice(0, 60))
    padded["positions"][[4, 20, 59]] = -1
    padded["token_row"][[5, 59]] = -1
    live = torch.ones(60, dtype=torch.bool)
    live[[4, 5, 20, 59]] = False
    for chunks in (0, 3):
        got = run_rows(padded, **shape, max_chunks=chunks)
        assert torch.equal(got[live.to(DEV)], walked[:60][live.to(DEV)]) and not got[~live.to(DEV)].any()


def test_a_later_token_that_is_not_finite_touches_no_earlier_one():
    case = paged_case(torch.float32, nq=4, nkv=2, d=128, page=16, lengths=[300], queries=[300], seed=3)
    shape = dict(nq=4, nkv=2, d=128, scale=128 ** -0.5, window=None, max_chunks=0)
    before = run_rows(case, **shape)
    for cache, at, value in (("kc", 290, float("inf")), ("vc", 270, float("nan"))):
        page = case["tables"][0, at // 16]
        case[cache][page, :, at % 16] = value
    after = run_rows(case, **shape)
    assert torch.equal(before[:270], after[:270]) and after[270:].isnan().all()


@pytest.mark.parametrize("heads", [(2, 2, 64), (8, 1, 128)])
def test_many_single_tokens_give_the_bits_they_give_alone(heads):
    """More (token, kv head) pairs than one look of the CTAs that deal them out, single tokens and runs in turn."""
    nq, nkv, d = heads
    tokens = 40000 // nkv
    case = paged_case(torch.float32, nq=nq, nkv=nkv, d=d, page=16, lengths=[300, 40, 70, 290], queries=[1, 1, 1, 1], seed=d)
    g = torch.Generator().manual_seed(nq)
    rows = torch.arange(tokens, dtype=torch.int32) % 3
    rows[100:140], rows[1000:1003], rows[tokens - 5:] = 3, 3, 3                # long runs, and one of three
    limits = torch.tensor([300, 40, 70, 290])[rows.long()]
    picked = dict(case, token_row=rows.to(DEV), positions=(torch.rand(tokens, generator=g) * limits).int().to(DEV),
                  q=torch.randn(tokens, nq * d, generator=g).to(DEV))
    shape = dict(nq=nq, nkv=nkv, d=d, scale=d ** -0.5, window=None)
    walked = run_rows(picked, **shape, max_chunks=0)
    for at in (0, 96, 130, 990, tokens // 2, tokens - 60):
        part = some_rows(picked, slice(at, at + 60))
        assert torch.equal(run_rows(part, **shape, max_chunks=2), walked[at:at + 60]), at


def test_single_tokens_run_side_by_side():
    """Decoded tokens of many requests, whose chunks are walked: 32 of them take about as long as one (in line they would
    take 16 times as long)."""
    times = []
    for count in (1, 32):
        case = paged_case(torch.float32, nq=16, nkv=8, d=128, page=16, lengths=[250] * count, queries=[1] * count, seed=count)
        case = {name: value.to(DEV) if torch.is_tensor(value) else value for name, value in case.items()}
        call = lambda: run_rows(case, nq=16, nkv=8, d=128, scale=128 ** -0.5, window=None, max_chunks=0)
        call()
        best = float("inf")
        for _ in range(20):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(5):
                call()
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        times.append(best)
    assert times[1] < 5 * times[0], times
