"""The one-call bookkeeping of a decode step against the same step as single calls: positions, slots, lengths, tables,
copy-on-write of shared blocks, padding rows and exhaustion."""
import random

import pytest
import torch

from ml_framework_b200._lib import MlfError
from ml_framework_b200.serving.kv_cache import KVCacheBlockManager


def _pool(rng, blocks, bs):
    m = KVCacheBlockManager(blocks, bs, head_dim=2, num_layers=2, num_kv_heads=1, device="cpu", dtype=torch.float32)
    for i, c in enumerate(m.caches):
        c.copy_(torch.arange(c.numel(), dtype=torch.float32).view(c.shape) + i)
    for s in range(5):
        m.append_tokens(s, rng.randint(1, 3 * bs))
    m.fork(1, 10)                     # shares a possibly partial last block: the next append copies it
    m.fork(10, 11)
    m.allocate_blocks(2, 1)           # a reserved block beyond the tokens
    return m


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("bs", [1, 4, 16])
@pytest.mark.parametrize("spare", [0, 1, 40])
def test_same_as_single_calls(seed, bs, spare):
    probe = _pool(random.Random(seed), 400, bs)
    total = 400 - probe.free_blocks + spare
    a, b = _pool(random.Random(seed), total, bs), _pool(random.Random(seed), total, bs)
    ids = [11, 3, 1, 77, 10, 2]       # 77 is new to the pool
    rows, width, max_blocks = 8, 7, 64
    pos = [a.get_sequence_length(s) for s in ids]
    slots, done = [], len(ids)
    for i, s in enumerate(ids):
        t, _ = a.append_tokens(s, 1)
        if t is None:
            done = i
            break
        slots.append(int(t[0]))
    h = torch.full((2, rows), -9, dtype=torch.int64)
    h32 = torch.full((rows * (1 + width),), -9, dtype=torch.int32)
    got, top = b.append_decode(ids, max_blocks, rows, width, h[0], h[1], h32[:rows], h32[rows:])
    assert got == done and top == max(pos)
    assert h[0, :6].tolist() == pos and h[1, :done].tolist() == slots
    assert a.get_stats() == b.get_stats()
    assert all(torch.equal(x, y) for x, y in zip(a.caches, b.caches))
    assert all(a.get_sequence_blocks(s) == b.get_sequence_blocks(s) for s in ids[:done])
    if done == len(ids):
        table, lens = a.build_tables(ids, max_blocks)
        t = h32[rows:].view(rows, width)
        assert torch.equal(h32[:6], lens) and torch.equal(t[:6], table[:, :width])
        assert h[0, 6:].tolist() == [0, 0] and h[1, 6:].tolist() == [-1, -1] and h32[6:8].tolist() == [1, 1] and not t[6:].any()


def test_table_too_small_and_empty_batch():
    m = _pool(random.Random(0), 400, 1)
    h = torch.zeros(2, 2, dtype=torch.int64)
    h32 = torch.zeros(2 * 4, dtype=torch.int32)
    m.append_tokens(3, 5)
    with pytest.raises(MlfError):
        m.append_decode([3], 2, 1, 2, h[0], h[1], h32[:1], h32[2:])
    assert m.append_decode([], 2, 0, 2, h[0], h[1], h32[:1], h32[2:]) == (0, 0)
