"""Decode attention straight from the QKV product against the rotation, the cache write and the attention as launches of
their own: the same arithmetic in the same order, so outputs and cache are equal bit for bit at the same split."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native
from ml_framework_b200.ops.gemm import gemm

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


@pytest.mark.parametrize("B,Hq,Hkv", [(1, 32, 8), (13, 16, 4), (40, 8, 8)])
def test_behind_a_running_product(B, Hq, Hkv):
    """norm -> QKV product -> decode with early reads, back to back and with rows of its own in every round: lengths, tables
    and cached rows are read while the product runs, what the product writes is not. Each round is a token further."""
    torch.manual_seed(B)
    K, D, bs, rounds, pages = 4096, 128, 16, 5, 40
    width = (Hq + 2 * Hkv) * D
    cache = torch.randn(B * pages, 2, bs, Hkv, D, device="cuda").to(torch.bfloat16)
    table = torch.randperm(B * pages, device="cuda").to(torch.int32).view(B, pages)
    start = torch.randint(1, pages * bs - rounds, (B,), device="cuda")
    lens = [(start + r).to(torch.int32) for r in range(rounds)]
    slots = [table.gather(1, ((n.long() - 1) // bs)[:, None])[:, 0].long() * bs + (n.long() - 1) % bs for n in lens]
    xs = [torch.randn(B, K, device="cuda").to(torch.bfloat16) for r in range(rounds)]
    g = torch.rand(K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(width, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    qkv = torch.full((B, width), 7.0, device="cuda", dtype=torch.bfloat16)
    rows = [torch.empty_like(qkv) for _ in range(rounds)]
    a_cache, b_cache = cache.clone(), cache.clone()
    flags = _lib.EPI_ACCUM | _lib.EPI_B_STATIC
    got = []
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000)
    for r in range(rounds):
        h, _, _ = native.norm_fwd(xs[r], g, None, 1e-5, True, want_stats=False, zero=qkv)
        gemm(h, w, out=qkv, flags=flags)
        got.append(native.paged_decode_rope(qkv, a_cache, table, lens[r], slots[r], Hq, Hkv, pages * bs, 500000.0, inputs_static=True))
        rows[r].copy_(qkv)                   # an ordinary launch: the early reads of the next round start behind it
    torch.cuda.synchronize()
    for r in range(rounds):
        rot = rows[r].clone()
        native.rope_kv_write_(rot, lens[r].long() - 1, slots[r], b_cache, Hq, Hkv, 500000.0)
        want = native.paged_decode(rot[:, :Hq * D].view(B, Hq, D), b_cache, table, lens[r], pages * bs, split_tokens=0)
        assert torch.equal(got[r], want), r
    assert torch.equal(a_cache, b_cache)
    # and the rows themselves are this round's product, as close as one sum of bf16 partial tiles is
    for r in range(rounds):
        xf = xs[r].float()
        hf = (xf * torch.rsqrt((xf * xf).mean(-1, keepdim=True) + 1e-5) * g.float()).to(torch.bfloat16).float()
        wantq = hf @ w.float().t()
        assert (rows[r].float() - wantq).pow(2).mean().sqrt() <= 2 ** -7 * wantq.pow(2).mean().sqrt()
    assert _lib.read_status() == 0
