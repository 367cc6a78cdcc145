"""Attention forward with more items (256 query rows of one head) than SMs, so that every CTA walks over several: ragged
last items, items without a second query tile, cached prefixes, NaN in, rows of the next sequence untouched."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native
from ml_framework_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu
D = 128


def _ref(q, k, v, B, Sq, Skv, causal):
    Hq, Hkv = q.shape[1], k.shape[1]
    qf = q.float().view(B, Sq, Hq, D).transpose(1, 2)
    kf, vf = (t.float().view(B, Skv, Hkv, D).transpose(1, 2).repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    s = (qf @ kf.transpose(-1, -2)) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(Sq, Skv, dtype=torch.bool, device=q.device).triu(1 + Skv - Sq), float("-inf"))
    return (s.softmax(-1) @ vf).transpose(1, 2).reshape(B * Sq, Hq, D), torch.logsumexp(s, -1)


def _inputs(B, Sq, Skv, Hq, Hkv, amp=1.0):
    torch.manual_seed(B * Sq + Skv)
    q = (torch.randn(B * Sq, Hq, D, device="cuda") * amp).to(torch.bfloat16)
    k, v = (torch.randn(B * Skv, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    return q, k, v


# 160 - 1500 items on 148 SMs; Sq around the tiles of 32 (a warp's rows), 128 (a query tile) and 256 (an item)
@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal,amp", [
    (5, 256, 256, 32, 8, True, 1.0), (5, 257, 257, 32, 8, True, 1.0), (5, 383, 383, 32, 8, True, 1.0), (3, 700, 700, 80, 16, True, 1.0),
    (4, 512, 512, 40, 40, False, 1.0), (4, 289, 289, 40, 40, False, 4.0), (2, 1025, 1025, 40, 8, True, 4.0),
    (5, 31, 541, 32, 8, True, 1.0), (5, 128, 640, 32, 8, True, 1.0), (3, 160, 800, 64, 8, True, 4.0), (160, 1, 130, 4, 1, True, 1.0)])
def test_items_per_cta(B, Sq, Skv, Hq, Hkv, causal, amp):
    q, k, v = _inputs(B, Sq, Skv, Hq, Hkv, amp)
    ref, ref_lse = _ref(q, k, v, B, Sq, Skv, causal)
    if Sq == Skv:
        out, lse = native.flash_fwd(q, k, v, B, Sq, causal=causal)
        # scores of up to 4 * 11.3 sigma in fp32: 1e-5 of the largest, and the sum of 2^-9-rounded weights never enters
        assert (lse - ref_lse).abs().max() < 1e-3
    else:
        out = native.flash_fwd_prefix(q, k, v, B, Sq, Skv, causal=causal)
    # P and the result are rounded to bf16 (2^-9 relative each), independently per element
    assert (out.float() - ref).norm() <= 5e-3 * ref.norm()
    assert (out.float() - ref).abs().max() <= 2e-2 * ref.abs().max()
    assert _lib.read_status() == 0


def test_output_rows_keep_to_their_buffer():
    """Wider row pitch than the heads need, and rows past the batch: neither is written."""
    B, S, H = 3, 300, 64
    q, k, v = _inputs(B, S, S, H, 8)
    buf = torch.full((B * S + 256, H * D + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    rc = _lib.get().mlf_flash_fwd_prefix(*(native._p(t) for t in (q, k, v, buf)), None, B, S, S, H, 8, *(native.C.c_longlong(n) for n in (
        H * D, 8 * D, 8 * D, H * D + 64)), native.C.c_float(D ** -0.5), 1, native._st())
    assert rc == 0
    want = native.flash_fwd(q, k, v, B, S, causal=True, want_lse=False)[0].view(B * S, -1)
    assert torch.equal(buf[:B * S, :H * D], want)
    assert (buf[B * S:] == 7).all() and (buf[:, H * D:] == 7).all()


def test_nan_key_reaches_every_row_that_sees_it():
    """A NaN in one key must not be lost in the exponentials, whichever pipe they run on."""
    B, S, H = 1, 256, 2
    q, k, v = _inputs(B, S, S, H, H)
    for pos in range(0, 64):
        kk = k.clone()
        kk[pos, 0, 5] = float("nan")
        out, _ = native.flash_fwd(q, kk, v, B, S, causal=True)
        bad = ~torch.isfinite(out.float()).all(-1)
        assert bad[pos:, 0].all() and not bad[:pos].any() and not bad[:, 1].any(), pos


def test_beside_a_kernel_that_holds_sms():
    """The items of CTAs that find no place beside another stream's kernel go to those that run: as many rounds as before, and
    not twice as many because some CTAs start when the others have ended."""
    B, S, H = 4, 2048, 16
    q, k, v = _inputs(B, S, S, H, H)
    a, o = torch.randn(8192, 8192, device="cuda").to(torch.bfloat16), torch.empty(8192, 8192, dtype=torch.bfloat16, device="cuda")
    side, reps, outs = torch.cuda.Stream(), 8, []

    def run(beside):
        torch.cuda.synchronize()
        e = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
        if beside:
            with torch.cuda.stream(side):
                gemm(a, a, out=o, tile_n=128, max_ctas=8)            # 15 ms on eight SMs
                e[2].record()
            torch.cuda._sleep(1_000_000)                             # until it holds them
        e[0].record()
        outs[:] = [native.flash_fwd(q, k, v, B, S)[0] for _ in range(reps)]
        e[1].record()
        torch.cuda.synchronize()
        assert not beside or e[1].elapsed_time(e[2]) > 0             # it held them to the end
        return e[0].elapsed_time(e[1]) / reps, outs[0]

    run(False)
    alone, want = min((run(False) for _ in range(3)), key=lambda r: r[0])
    beside, got = min((run(True) for _ in range(3)), key=lambda r: r[0])
    # 140 of 148 SMs: 1.06 times the time, and the last round's items; CTAs that wait for a place cost 1.7 times
    assert torch.equal(got, want) and beside <= 1.35 * alone, (alone, beside)
