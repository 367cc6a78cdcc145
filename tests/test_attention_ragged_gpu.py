"""Attention gradients at sequence lengths that are no multiple of four (the statistics' rows are padded) and around the
128-token tiles, for several sequences and heads so that every row of the statistics has its own alignment."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [128, 129, 130, 131, 255, 257, 383, 515, 777])
@pytest.mark.parametrize("B,Hq,Hkv,causal", [(3, 2, 1, True), (2, 3, 3, False)])
def test_gradients_ragged(S, B, Hq, Hkv, causal):
    torch.manual_seed(S)
    D = 128
    q, do = (torch.randn(B * S, Hq, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B * S, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    # whatever the scratch buffer held before must not matter
    native.scratch("flash_bwd", 1 << 24, q.device).view(torch.float32).fill_(float("nan"))
    o, lse = native.flash_fwd(q, k, v, B, S, causal=causal)
    dq, dk, dv = native.flash_bwd(q, k, v, o, do, lse, B, S, causal=causal)
    ref = [t.float().view(B, S, -1, D).transpose(1, 2).requires_grad_() for t in (q, k, v)]
    kk, vv = (t.repeat_interleave(Hq // Hkv, 1) for t in ref[1:])
    s = (ref[0] @ kk.transpose(-1, -2)) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ((s.softmax(-1) @ vv).transpose(1, 2).reshape(B * S, Hq, D) * do.float()).sum().backward()
    for got, want in zip((o, dq, dk, dv), (None, ref[0].grad, ref[1].grad, ref[2].grad)):
        assert torch.isfinite(got).all()
        if want is None:
            continue
        w = want.transpose(1, 2).reshape(got.shape)
        # P, dS and the results are rounded to bf16 (2^-9 relative each, O enters delta rounded): 1.5 % of the norm
        assert (got.float() - w).norm() <= 1.5e-2 * w.norm()
    assert _lib.read_status() == 0
