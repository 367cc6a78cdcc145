"""Vectorised element-wise kernels at their edges: remainders of the vector width, unaligned buffers, in place."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4099, 1 << 20, 303104 * 4 + 5])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("accumulate", [False, True])
def test_cast(n, shift, accumulate):
    torch.manual_seed(n)
    src = torch.randn(n + shift, device="cuda")[shift:]
    buf = torch.randn(n + shift + 8, device="cuda").to(torch.bfloat16)
    guard = buf.clone()
    out = buf[shift:shift + n]
    want = (src + out.float() if accumulate else src).to(torch.bfloat16)
    native.cast_f32_to_bf16(src, out, accumulate)
    assert torch.equal(out, want)
    assert torch.equal(buf[:shift], guard[:shift]) and torch.equal(buf[shift + n:], guard[shift + n:])


@pytest.mark.parametrize("T,D", [(1, 8), (37, 264), (513, 1024)])
@pytest.mark.parametrize("shift", [0, 1])
def test_embedding_gradient(T, D, shift):
    torch.manual_seed(T)
    V = 50
    ids = torch.randint(0, V, (T,), device="cuda")
    ids[0] = V + 3                                    # outside the table: skipped
    dout = torch.randn(T, D, device="cuda").to(torch.bfloat16)
    dw = torch.zeros(V * D + shift, device="cuda")[shift:].view(V, D)
    native.embedding_bwd(dout, ids, V, dw)
    want = torch.zeros(V, D, device="cuda", dtype=torch.float64).index_add_(0, ids[1:], dout[1:].double())
    # fp32 sums of up to T / V + a few terms of order 1 in any order
    assert ((dw.double() - want).abs() <= 1e-5 * (1 + want.abs())).all()


@pytest.mark.parametrize("T", [1, 31, 1000])
@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (2, 1), (8, 2), (5, 5)])
@pytest.mark.parametrize("inverse", [False, True])
def test_rope_qkv(T, Hq, Hkv, inverse):
    torch.manual_seed(T)
    W = (Hq + 2 * Hkv) * 128
    wide = torch.randn(T, W + 16, device="cuda").to(torch.bfloat16)
    src = wide[:, 8:8 + W]
    pos = torch.randint(0, 5000, (T,), device="cuda")
    want = src.clone()
    native.rope_(want[:, :Hq * 128].view(T, Hq, 128), pos, 500000.0, inverse)
    native.rope_(want[:, Hq * 128:(Hq + Hkv) * 128].view(T, Hkv, 128), pos, 500000.0, inverse)
    before = wide.clone()
    got = native.rope_qkv(src, pos, Hq, Hkv, 500000.0, inverse)
    assert torch.equal(got, want)                     # one statement of the angle and of the rotation, roundings and all
    assert torch.equal(got[:, (Hq + Hkv) * 128:], src[:, (Hq + Hkv) * 128:]) and torch.equal(wide, before)
    native.rope_qkv(src, pos, Hq, Hkv, 500000.0, inverse, out=src)
    assert torch.equal(src, got) and torch.equal(wide[:, :8], before[:, :8]) and torch.equal(wide[:, 8 + W:], before[:, 8 + W:])
    assert _lib.read_status() == 0


@pytest.mark.parametrize("V", [7, 4095, 8184, 8191, 8192, 8199, 16400])
def test_cross_entropy_around_two_vectors_per_thread(V):
    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    logits = (torch.randn(9, ld, device="cuda") * 3).to(torch.bfloat16)
    logits[2, : V // 2] = -torch.inf
    tg = torch.randint(V // 2, V, (9,), device="cuda")
    tg[4] = -100
    z = logits[:, :V].double()
    lse = z.logsumexp(-1)
    keep = tg >= 0
    want = torch.where(keep, lse - z.gather(1, tg.clamp(min=0)[:, None])[:, 0], 0.0)
    grad = (z.softmax(-1) - torch.nn.functional.one_hot(tg.clamp(min=0), V)) * keep[:, None] * 0.25
    loss, _ = native.cross_entropy_(logits, tg, V, grad_scale=0.25)
    # fp32 sums of V terms with exponentials of 2^-21 each; one rounding of the gradient to bf16
    assert ((loss.double() - want).abs() <= 1e-5 * (1 + want.abs())).all()
    assert ((logits[:, :V].double() - grad).abs() <= 2 ** -8 * grad.abs() + 1e-6).all()
    assert not logits[:, V:].any()
    assert _lib.read_status() == 0


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("extra", [0, 5])
def test_packed_attention_takes_a_longer_position_buffer(dtype, extra):
    from ml_framework_b200.ops import functional as Fm
    torch.manual_seed(0)
    B, S, Hq, Hkv = 2, 48, 4, 2
    base = torch.randn(B * S, (Hq + 2 * Hkv) * 128, device="cuda").to(torch.bfloat16)
    pos = torch.cat([torch.arange(S).repeat(B), torch.full((extra,), 7)]).to("cuda", dtype)
    outs = []
    for p in (None, pos):
        qkv = base.clone().requires_grad_()
        o = Fm.attention_packed(qkv, B, S, Hq, Hkv, 128, True, 10000.0, p)
        o.backward(torch.ones_like(o))
        outs.append((o.detach(), qkv.grad))
    # forward bit for bit; dQ is summed over key tiles in any order before it is rounded to bf16
    assert torch.equal(outs[0][0], outs[1][0])
    assert ((outs[0][1].float() - outs[1][1].float()).abs() <= 2 ** -7 * outs[0][1].float().abs() + 2 ** -12).all()
    with pytest.raises(AssertionError):
        Fm.attention_packed(base, B, S, Hq, Hkv, 128, True, 10000.0, pos[:B * S - 1])
