"""Decode attention straight from the QKV product against the rotation, the cache write and the attention as launches of
their own: the same arithmetic in the same order, so outputs and cache are equal bit for bit at the same split."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (4, 2), (16, 4), (8, 1)])
@pytest.mark.parametrize("split", [0, 128, 384])
@pytest.mark.parametrize("bs,static", [(16, False), (16, True), (24, True)])
def test_same_as_separate_launches(Hq, Hkv, split, bs, static):
    torch.manual_seed(Hq * 10 + Hkv)
    # chunk and split edges: the newest token alone, first / last of a 64-token chunk, of a split, of a page
    lens = [1, 2, 16, 17, 63, 64, 65, 128, 129, 385, 640, 1, 1000]
    B, D = len(lens), 128
    pages = [(n + bs - 1) // bs for n in lens]
    nb = sum(pages) + 1
    perm = torch.randperm(nb - 1) + 1
    table = torch.zeros(B, max(pages), dtype=torch.int32)
    used = 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[used:used + n]
        used += n
    slots = torch.tensor([int(table[i, (n - 1) // bs]) * bs + (n - 1) % bs for i, n in enumerate(lens)])
    slots[11] = -1                                    # a padding row: attends to its own token, writes nothing
    cache = torch.randn(nb, 2, bs, Hkv, D, device="cuda").to(torch.bfloat16)
    wide = torch.randn(B, (Hq + 2 * Hkv) * D + 64, device="cuda").to(torch.bfloat16)
    qkv = wide[:, :(Hq + 2 * Hkv) * D]
    table, slots = table.cuda(), slots.cuda()
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    a_cache, b_cache, rot = cache.clone(), cache.clone(), qkv.clone()
    native.rope_kv_write_(rot, sl.long() - 1, slots, a_cache, Hq, Hkv, 500000.0)
    # the separate path finds the padding row's key and value in the cache; its block is nobody else's
    pad = int(table[11, 0])
    probe = a_cache.clone()
    probe[pad, 0, 0] = rot[11, Hq * D:(Hq + Hkv) * D].view(Hkv, D)
    probe[pad, 1, 0] = rot[11, (Hq + Hkv) * D:].view(Hkv, D)
    want = native.paged_decode(rot[:, :Hq * D].view(B, Hq, D), probe, table, sl, max(lens), split_tokens=split)
    got = native.paged_decode_rope(qkv, b_cache, table, sl, slots, Hq, Hkv, max(lens), 500000.0, split_tokens=split,
                                   inputs_static=static)
    assert torch.equal(got, want)
    assert torch.equal(a_cache, b_cache)
    assert _lib.read_status() == 0
