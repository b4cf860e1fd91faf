"""Thresholds of top-k and top-p at vocabularies where a CTA's part of the row is ragged, empty or too long for shared memory:
the tokens against the plain rules, and ties at the k-th score over the parts' boundaries."""

import pytest
import torch

from test_kernels_gpu import DEV, k, pack, plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [1, 3, 5, 29, 4097, 151936, 520001])
def test_thresholds(vocab):
    generator = torch.Generator().manual_seed(vocab)
    rows = [(0.8, 7, 1.0, 1, 0), (0.8, 1, 1.0, 2, 0), (1.1, vocab - 1, 1.0, 3, 1), (0.8, 0, 0.9, 4, 2), (0.8, 50, 0.5, 5, 3),
            (0.8, 0, 1e-6, 6, 4), (0.0, 5, 0.5, 7, 5), (0.7, 0, 1.0, 8, 6)]
    logits = torch.randn(len(rows), vocab + 1, generator=generator)[:, 1:] * 2.0       # rows off the 16-byte boundary too
    got = k().sample_rows(logits.to(DEV), pack(rows)).cpu().tolist()
    aligned = k().sample_rows(logits.contiguous().to(DEV), pack(rows)).cpu().tolist()
    want = [plain.sample(logits[i], *rows[i]) for i in range(len(rows))]
    assert got == want and aligned == want


@pytest.mark.parametrize("at", [0, 19, 20, 39, 150])
def test_ties_stay_by_token_id_across_parts(at):
    vocab, wanted = 160, 5                                     # parts of 20 tokens
    logits = torch.full((1, vocab), -30.0)
    equals = [i for i in range(at, vocab, 3)][:7]
    logits[0, equals] = 1.0
    logits[0, (at + 1) % vocab] = 2.0                          # one above: wanted - 1 of the equals stay
    seen = {k().sample_rows(logits.to(DEV), pack([(50.0, wanted, 1.0, seed, 0)])).item() for seed in range(200)}
    kept = set(equals[:wanted - 1]) | {(at + 1) % vocab}
    if (at + 1) % vocab in equals:
        kept = {(at + 1) % vocab} | set([i for i in equals if i != (at + 1) % vocab][:wanted - 1])
    assert seen == kept if len(equals) >= wanted - 1 else kept <= seen
