"""Rotary embedding and cache write of packed rows against the same two steps one after the other (bit for bit: the angles
and rotations are the same statements): 16- and 8-byte aligned rows, few tokens (heads split over several warps) and many,
head counts that are no multiple of four, skipped slots."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu
D, PAGE = 128, 16


@pytest.mark.parametrize("T", [1, 7, 8, 9, 37, 300, 2369])
@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (5, 3), (32, 8), (40, 40)])
@pytest.mark.parametrize("pad,offset", [(0, 0), (4, 0), (8, 4)])      # elements: 8-byte rows, an 8-byte base
def test_matches_separate_steps(T, Hq, Hkv, pad, offset):
    torch.manual_seed(T + Hq)
    W = (Hq + 2 * Hkv) * D
    buf = torch.randn(T * (W + pad) + 16, device="cuda").to(torch.bfloat16)
    qkv = buf[offset:offset + T * (W + pad)].view(T, W + pad)[:, :W]
    want = qkv.clone()
    pos = torch.randint(0, 9000, (T,), device="cuda")
    blocks = (T + PAGE - 1) // PAGE + 1
    slots = torch.randperm(blocks * PAGE, device="cuda")[:T]
    slots[T // 2] = -1
    cache = torch.full((blocks, 2, PAGE, Hkv, D), 3.0, dtype=torch.bfloat16, device="cuda")
    want_cache = cache.clone()
    before = buf.clone()
    native.rope_kv_write_(qkv, pos, slots, cache, Hq, Hkv, 5e5)
    native.rope_(want[:, :(Hq + Hkv) * D].view(T, Hq + Hkv, D), pos, 5e5)
    flat = want_cache.permute(1, 0, 2, 3, 4)
    ok = slots >= 0
    at = (slots[ok] // PAGE, slots[ok] % PAGE)
    flat[0][at] = want[ok, Hq * D:(Hq + Hkv) * D].view(-1, Hkv, D)
    flat[1][at] = want[ok, (Hq + Hkv) * D:].view(-1, Hkv, D)
    assert torch.equal(qkv, want) and torch.equal(cache, want_cache)
    rest = torch.ones_like(buf, dtype=torch.bool)
    rest[offset:offset + T * (W + pad)].view(T, W + pad)[:, :W] = False
    assert torch.equal(buf[rest], before[rest])
    assert _lib.read_status() == 0
