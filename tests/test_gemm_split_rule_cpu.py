"""Into how many parts a CTA-pair product splits K: never more than the coarsest count that pays."""
import pytest

from ml_framework_b200 import _lib


def _by_rounds(tiles, K, pairs):
    """(parts, rounds) by the number of rounds alone: each finer count has to save a tenth of them."""
    best, parts, kb = float(-(-tiles // pairs)), 1, -(-K // 64)
    for ks in range(2, 9):
        if kb // ks < 8:
            break
        cost = float(-(-tiles * ks // pairs)) / ks
        if cost < best * 0.9:
            best, parts = cost, ks
    return parts, best


@pytest.mark.parametrize("pairs", [74, 72, 66, 8])
@pytest.mark.parametrize("K", [512, 1000, 1024, 2560, 4096, 8192, 50304])
def test_parts_are_bounded_and_pay(pairs, K):
    split = _lib.get().mlf_gemm_k_splits
    for tiles in range(1, 8 * pairs + 1):
        got = split(tiles, K, pairs)
        parts, _ = _by_rounds(tiles, K, pairs)
        assert 1 <= got <= parts
        if got > 1:
            rest = tiles % pairs
            whole = -(-tiles // pairs) - (0.2 if 0 < rest and 2 * rest <= pairs else 0.0)
            assert float(-(-tiles * got // pairs)) / got < 0.8 * whole
            assert -(-K // 64) // got >= 8


@pytest.mark.parametrize("tiles,parts", [(99, 1), (100, 1), (105, 1), (108, 1), (112, 1), (116, 1), (128, 1), (56, 1), (75, 6), (96, 3), (8, 8)])
def test_counts_on_74_pairs(tiles, parts):
    assert _lib.get().mlf_gemm_k_splits(tiles, 8192, 74) == parts
