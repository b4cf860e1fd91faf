"""Kernels whose shared memory depends on the sizes, launched from two threads with sizes far apart: neither thread's launch
may meet the other's limit."""

import threading

import pytest
import torch

from tinyvllm_b200.ops import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def sampling(vocab):
    from test_kernels_gpu import pack

    logits = torch.randn(4, vocab, device=DEV)
    packed = pack([(0.8, 5, 1.0, 1, 0)] * 4)
    return lambda: kernels.sample_rows(logits, packed)


def few_rows(k):
    a, w = torch.randn(2, k, device=DEV), torch.randn(24, k, device=DEV)
    return lambda: kernels.gemm_nt_simt(a, w)


def retention(dim):
    tokens, heads = 160, 2
    per = heads * dim
    proj = torch.randn(tokens, 3 * per, device=DEV)
    state, decay = torch.zeros(1, heads, dim, dim, device=DEV), torch.full((heads,), 0.97, device=DEV)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts, slots, rows = i32(0, tokens), i32(0), torch.zeros(tokens, dtype=torch.int32, device=DEV)
    positions = torch.arange(tokens, dtype=torch.int32, device=DEV)

    def call():
        state.zero_()
        return kernels.retention(proj, q_at=0, k_at=per, v_at=2 * per, g_at=None, heads=heads, dim=dim, vdim=dim, decay=decay,
                                 state=state, row_starts=starts, state_slots=slots, token_row=rows, positions=positions,
                                 segment=64)
    return call


@pytest.mark.parametrize("make,small,large", [(sampling, 100, 400000), (few_rows, 128, 12000), (retention, 8, 256)])
def test_two_threads_with_sizes_far_apart(make, small, large):
    calls = [make(small), make(large)]
    want = [call() for call in calls]
    torch.cuda.synchronize()
    failures = []

    def work(call, want):
        try:
            for _ in range(1500):
                got = call()
            torch.cuda.synchronize()
            assert torch.equal(got, want)
        except Exception as failure:                       # noqa: BLE001 (raised in the test's own thread below)
            failures.append(failure)

    threads = [threading.Thread(target=work, args=pair) for pair in zip(calls, want)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not failures, failures
