"""Thresholds of top-k and top-p at vocabularies where a CTA's part of the row is ragged, empty or too long for shared memory:
the tokens against the plain rules, and ties at the k-th score over the parts' boundaries; batches whose greedy rows have a
launch of their own."""

import functools

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


VOCAB = 151936
KINDS = {"greedy": [(0.0, 0, 1.0)], "sampled": [(0.8, 50, 1.0), (0.8, 0, 0.95), (0.7, 40, 0.9), (1.0, 0, 1.0)],
         "mixed": [(0.0, 0, 1.0), (0.8, 50, 1.0), (0.0, 7, 0.5), (0.8, 0, 0.95)]}


@functools.cache
def many_logits():
    return torch.randn(75, VOCAB, generator=torch.Generator().manual_seed(75)) * 2.0


@functools.cache
def wanted(row, temperature, top_k, top_p):
    return plain.sample(many_logits()[row], temperature, top_k, top_p, row, 3)


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("count", [37, 38, 48, 64, 75])
def test_larger_batches_follow_the_plain_rules(count, kind):
    rows = [(*KINDS[kind][i % len(KINDS[kind])], i, 3) for i in range(count)]
    got = k().sample_rows(many_logits()[:count].to(DEV), pack(rows)).cpu().tolist()
    assert got == [wanted(i, *row[:3]) for i, row in enumerate(rows)]


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("count", [37, 64])
def test_what_follows_the_sampling_sees_its_tokens(count, kind):
    """A captured step as the decode graphs have it: sampling, then a copy of the tokens.  The copy is compared, with
    logits that change from replay to replay."""
    rows = [(*KINDS[kind][i % len(KINDS[kind])], i, 3) for i in range(count)]
    packed, every = pack(rows), many_logits().to(DEV)
    logits, tokens = torch.zeros(count, VOCAB, device=DEV), torch.zeros(count, dtype=torch.int32, device=DEV)
    copy = torch.zeros_like(tokens)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        k().sample_rows(logits, packed, out=tokens)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            k().sample_rows(logits, packed, out=tokens)
            copy.copy_(tokens)
        for shift in range(30):
            logits.copy_(every[:count].roll(shift + 1, 0))
            graph.replay()
            seen = copy.clone()
            assert torch.equal(seen, k().sample_rows(logits, packed)), shift
            if kind == "greedy":
                assert torch.equal(seen, logits.argmax(1).int()), shift
