"""Tokens per split of paged decode attention, from the pairs of sequence and KV head and the length bound."""
import pytest

from ml_framework_b200.ops.native import _decode_split


@pytest.mark.parametrize("sms", [148, 132, 1])
def test_bounds(sms):
    for pairs in (1, 8, 104, 160, 222, 223, 256, 444, 445, 512, 1024, 4096):
        for length in (1, 127, 128, 129, 512, 1024, 1025, 4096, 131072):
            tokens = _decode_split(pairs, length, sms)
            splits = -(-length // tokens)
            assert 1 <= tokens <= length and (splits == 1 or tokens >= 64)
            # within three rounds of resident CTAs, one round where that leaves at most 1400 tokens to a split
            assert splits * pairs <= max(pairs, 9 * sms)
            if splits > 1 and -(-length // max(1, 3 * sms // pairs)) <= 1400:
                assert splits * pairs <= 3 * sms


@pytest.mark.parametrize("pairs,length,splits", [
    # resident at once
    (512, 1024, 1), (384, 1024, 1), (104, 4096, 4), (128, 4096, 3), (64, 8192, 6), (2048, 2048, 1), (960, 1024, 1), (8, 1024, 8),
    (296, 2048, 1), (444, 2048, 1),
    # two rounds, three rounds
    (128, 8192, 6), (160, 4096, 5), (224, 2048, 3), (256, 2048, 3), (256, 4096, 3),
    (256, 8192, 5), (512, 4096, 2), (448, 8192, 2), (512, 2048, 2)])
def test_long_sequences_are_split(pairs, length, splits):
    """A sequence of 8192 tokens beside short ones, on 256 pairs, took 124 us in one split and 42 in five."""
    assert -(-length // _decode_split(pairs, length, 148)) == splits
