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


@pytest.mark.parametrize("D,rms", [(2048, False), (2048, True), (4096, False), (4096, True)])
@pytest.mark.parametrize("rows", [1, 295, 296, 297, 591, 592, 593, 1183, 1185, 2371])
def test_norm_rows_per_cta(D, rms, rows):
    """Whole-CTA rows around one, two and several groups of rows per CTA (148 SMs: 296 CTAs), the buffer cleared beside."""
    torch.manual_seed(rows)
    x = torch.randn(rows, D, device="cuda").to(torch.bfloat16) + 0.5
    g, b = (torch.randn(D, device="cuda").to(torch.bfloat16) for _ in range(2))
    zero = torch.full((rows, 64), 5.0, dtype=torch.bfloat16, device="cuda")
    y, mean, rstd = native.norm_fwd(x, g, None if rms else b, 1e-5, rms, zero=zero)
    xd = x.double()
    mu = torch.zeros(rows, 1, dtype=torch.float64, device="cuda") if rms else xd.mean(-1, keepdim=True)
    r = ((xd - mu).square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    want = (xd - mu) * r * g.double() + (0 if rms else b.double())
    assert ((rstd.double() - r[:, 0]) / r[:, 0]).abs().max() < 1e-5          # fp32 sums of 4096 squares
    assert rms or (mean.double() - mu[:, 0]).abs().max() < 1e-5
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()      # one rounding to bf16
    assert (zero == 0).all() and _lib.read_status() == 0
