"""The tile shares of the batched decode attention (csrc/attn_decode.cu, balanced grid) where the engine chooses the split length: as in
test_attn_partition.py, and Q no less than the longest sequence where that has at most four tiles."""
import random

from test_attn_partition import TILE, check, partition

WHOLE = 4


def engine_split_len(lens, split_len):
    """The split length with which the general law gives the engine's Q."""
    longest = max((length + TILE - 1) // TILE for length in lens)
    return max(split_len, longest * TILE) if longest <= WHOLE else split_len


def engine_partition(lens, groups, n_splits, split_len):
    return partition(lens, groups, n_splits, engine_split_len(lens, split_len))


def test_every_tile_once_and_pieces_fit_the_slots():
    rng = random.Random(11)
    for _ in range(400):
        max_len = rng.choice([1, 64, 65, 200, 256, 257])
        lens = [rng.randint(1, max_len) for _ in range(rng.randint(2, 256))]
        if rng.random() < 0.5:
            lens[rng.randrange(len(lens))] = max_len
        split_len = rng.choice([32, 64, 128, 256])
        n_splits = max(1, (max(lens) + split_len - 1) // split_len)
        check(lens, rng.choice([1, 3, 55, 111, 444]), n_splits, engine_split_len(lens, split_len))


def test_short_sequences():
    # whole where the even share is smaller than a sequence, cut on the multiples of Q where it is larger
    assert len(engine_partition([200] * 5, 55, 4, 128)) == 5 and len(partition([200] * 5, 55, 4, 128)) == 10
    assert len(engine_partition([256] * 13, 55, 4, 128)) == 13
    assert len(engine_partition([208] * 96, 55, 4, 128)) == 96 + 41  # Q = 7


def test_long_sequences_have_even_shares():
    assert engine_partition([257] * 5, 55, 3, 128) == partition([257] * 5, 55, 3, 128)
    # the even share (11 tiles) is larger than either split length
    assert engine_partition([1100] * 32, 55, 16, 128) == partition([1100] * 32, 55, 5, 256)
