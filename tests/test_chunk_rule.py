"""Which sequences of a step the chunked state scans take: a few long ones, whatever lies beside them; padding and small differences
of length decide nothing."""
import heapq
import random
from types import SimpleNamespace

import pytest

from gguf2bin_b200 import kernels

KINDS = [(0, 8, 256, 128), (2, 64, 64, 128), (2, 8, 257, 128), (1, 8, 128, 128), (0, 4, 64, 32), (1, 2, 32, 32)]


def plan_of(lens, kind, pad=0):
    return kernels.scan_plan(SimpleNamespace(q_lens=[*lens, pad] if pad else lens, padded=bool(pad)), kind)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("beside", [[], [1] * 30, [7, 60, 3], [1] * 8 + [50]])
def test_a_long_prompt_goes_in_chunks_whatever_lies_beside_it(kind, beside):
    for lens in ([*beside, 2048], [2048, *beside]):
        over, chunks, padding, chain = plan_of(lens, kind)
        assert 64 <= over < 2048 and (chunks, padding, chain) == (32, False, bool(beside))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("lens", [[1, 2], [64], [33, 64, 2], [64] * 40])
def test_no_prompt_of_a_chunk_or_less(kind, lens):
    assert plan_of(lens, kind) == (kernels.NO_CHUNKS, 0, False, True) == plan_of(lens, kind, pad=30)


@pytest.mark.parametrize("kind", KINDS[:4])
def test_large_batches_keep_the_gpu_busy_a_token_after_a_token(kind):
    assert plan_of([200] * 40, kind)[0] == kernels.NO_CHUNKS


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rest", [[], [20], [1, 1, 300]])
def test_a_bucket_of_lengths_has_one_plan(kind, rest):
    """A prompt of 1 to 63 tokens less than a multiple of 64, with padding that fills it up, is one shape: one graph."""
    for top in (128, 320, 2048):
        free = sum(rest) % 64
        plans = {plan_of([n, *rest], kind, pad=(-n - free) % 64) for n in range(top - 63, top) if (n + free) % 64}
        if not rest:
            assert len(plans) <= 2 and (top < 320 or len(plans) == 1)      # at most where the rule changes its mind inside a bucket
        assert all(p[0] in (64, kernels.NO_CHUNKS) or p[0] % 32 == 0 for p in plans)


@pytest.mark.parametrize("kind", KINDS)
def test_padding_decides_nothing(kind):
    for lens in ([100], [97], [500, 20], [130, 130], [2000]):
        bare = plan_of(lens, kind)
        for pad in (1, 28, 63):
            over, chunks, padding, chain = plan_of(lens, kind, pad)
            assert (over, chain) == (bare[0], bare[3])
            assert (chunks, padding) == ((bare[1] + 1, True) if bare[1] else (0, False))


def test_every_chunk_is_counted():
    for kind in KINDS:
        over, chunks, _, chain = plan_of([1501, 900, 400, 130, 64, 5], kind)
        if over != kernels.NO_CHUNKS:
            taken = [n for n in (1501, 900, 400, 130, 64, 5) if n > over]
            assert chunks == sum(-(-n // 64) for n in taken) and chain and taken[0] == 1501


def plain_chain_us(lens, n_seqs, mode, heads, cols, dim):
    lanes = 8
    while lanes * 16 < dim:
        lanes *= 2
    while lanes < 32 and n_seqs * heads * cols * lanes * 2 <= 76800:
        lanes *= 2
    padded = -(-dim // (4 * lanes)) * 4 * lanes
    tile = 16 if padded <= 128 else 8 if padded <= 256 else 4
    blocks = heads * -(-cols // (128 // lanes))
    per_sm = min(16, 227 * 1024 // (4 * tile * (4 * padded + 2 * (128 // lanes + 2) + 128) + 1024))
    first, more = {(1, 8): (0.42, 0.04), (1, 16): (0.33, 0.03), (1, 32): (0.31, 0.03)}.get(
        (mode, lanes), {8: (0.25, 0.045), 16: (0.20, 0.03), 32: (0.15, 0.03)}[lanes])
    token = first + more * min(blocks * len(lens) / 148, per_sm)
    free, end = [(0.0, 148 * per_sm)], 0.0   # slots of the GPU by when they come free
    for n in lens:
        left = blocks
        while left:
            at, slots = heapq.heappop(free)
            take = min(slots, left)
            left -= take
            if slots > take:
                heapq.heappush(free, (at, slots - take))
            heapq.heappush(free, (at + n * token, take))
            end = max(end, at + n * token)
    return 6.0 + end


def plain_rule(q_lens, mode, heads, cols, dim):
    step = 32
    classes = [-(-n // step) if n > 8 else 0 for n in q_lens]
    lens = [(c - 0.5) * step if c else 4.0 for c in classes]
    wide = heads * -(-cols // 64) * 64 * dim
    link, token = (0.04 + 0.0006 * dim, heads * cols * dim * 0.95e-6) if mode == 1 else (0.0, wide * 3.3e-7)
    best, over = 0.95 * plain_chain_us(lens, len(lens), mode, heads, cols, dim), None
    cuts = sorted({c for c in classes if c * step > 64})
    if len(cuts) > 8:
        cuts = [cuts[i * len(cuts) // 8] for i in range(8)]
    for cut in cuts:
        long = [-(-c * step // 64) * 64 for c in classes if c >= cut]
        short = [n for n, c in zip(lens, classes) if c < cut]
        us = 22.0 + max(max(long) * link, sum(long) * token)
        if short and us < best:
            us += plain_chain_us(short, len(lens), mode, heads, cols, dim)
        if us < best:
            best, over = us, max(max((c * step for c in classes if c < cut), default=0), 64)
    return over


@pytest.mark.parametrize("kind", KINDS)
def test_the_rule_as_it_is_written(kind):
    """The estimates restated, for few and many sequences, ragged, equal and with single tokens among them."""
    rng = random.Random(sum(kind))
    for n in (1, 2, 5, 9, 17, 33, 64, 150):
        for most in (60, 400, 3000):
            for lens in ([rng.randint(1, most) for _ in range(n)], [most] * n, [rng.choice((1, 1, rng.randint(1, most))) for _ in range(n)]):
                assert kernels._scan_chunks_over(lens, *kind) == plain_rule(lens, *kind), lens
