"""Host side of a step: token ids converted and checked as a whole, and the attention's work list (no GPU)."""
import numpy as np
import pytest

from gguf2bin_b200.engine.step import StepError, attention_tiles, token_ids


@pytest.mark.parametrize("tokens", [[0], [1, 2, 310], (5, 7), [np.int64(3), np.int32(4)], np.array([1, 2]), [True, 2], [2.0, 3.7], range(4)])
def test_ids_that_are_taken(tokens):
    assert token_ids(tokens, 311).tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("tokens,bad", [([311], "311"), ([0, -1], "-1"), ([3, 2 ** 70], str(2 ** 70)), ((0, 400), "400"), (np.array([1, 999]), "999"),
                                        ([1.0, 311.5], "311.5"), ([5, -(2 ** 64), 311], str(-(2 ** 64)))])
def test_ids_outside_the_vocabulary_are_refused(tokens, bad):
    with pytest.raises(StepError, match=f"token id {bad} outside the vocabulary 0..310"):
        token_ids(tokens, 311)


@pytest.mark.parametrize("rows", [64, 128])
@pytest.mark.parametrize("q_lens,past", [([1], [0]), ([1, 1, 1], [5, 0, 200]), ([64, 130, 1], [0, 7, 999]), ([2048], [0]), ([200, 1, 63, 512], [64, 0, 1, 3])])
def test_work_list(q_lens, past, rows):
    tiles, t0 = [], 0
    for b, n in enumerate(q_lens):
        tiles += [(b, t0 + r, min(rows, n - r), past[b] + r) for r in range(0, n, rows)]
        t0 += n
    tiles.sort(key=lambda t: -(t[3] + t[2]))
    got = attention_tiles(q_lens, past, rows)
    assert got.dtype == np.int32 and got.tolist() == [list(t) for t in tiles]
