"""Attention backward into packed gradient rows: last warps of a sequence that are not whole, rows of the next sequence, rows
behind the batch and columns beside the heads stay what they are; scratch contents do not matter."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("B,S,Hq,Hkv,causal", [(1, 128, 1, 1, True), (3, 129, 2, 1, True), (2, 159, 2, 2, True), (2, 160, 2, 2, True), (2, 161, 2, 2, False),
                                               (2, 257, 3, 3, False), (2, 777, 4, 2, True), (2, 96, 2, 2, True)])
def test_packed_gradients(B, S, Hq, Hkv, causal):
    torch.manual_seed(S)
    T, W = B * S, (Hq + 2 * Hkv) * D
    q, do = (torch.randn(T, Hq, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(T, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    native.scratch("flash_bwd", 1 << 24, q.device).view(torch.float32).fill_(float("nan"))
    o, lse = native.flash_fwd(q, k, v, B, S, causal=causal)
    buf = torch.full((T + 64, W + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    d = buf[:T, :W]
    dq, dk, dv = (d[:, a * D:b * D].unflatten(1, (-1, D)) for a, b in ((0, Hq), (Hq, Hq + Hkv), (Hq + Hkv, Hq + 2 * Hkv)))
    native.flash_bwd(q, k, v, o, do, lse, B, S, causal=causal, dq=dq, dk=dk, dv=dv)
    ref = [t.double().view(B, S, -1, D).transpose(1, 2).requires_grad_() for t in (q, k, v)]
    kk, vv = (t.repeat_interleave(Hq // Hkv, 1) for t in ref[1:])
    s = (ref[0] @ kk.transpose(-1, -2)) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ((s.softmax(-1) @ vv).transpose(1, 2).reshape(T, Hq, D) * do.double()).sum().backward()
    for got, r in zip((dq, dk, dv), ref):
        want = r.grad.transpose(1, 2).reshape(got.shape)
        # P, dS, O and the result are rounded to bf16 (2^-9 each at most)
        assert (got.double() - want).norm() <= 6e-3 * want.norm()
    assert (buf[T:] == 7).all() and (buf[:, W:] == 7).all() and _lib.read_status() == 0
