"""Normalisation backward at every width: rows around one, two and more rounds of the CTAs, groups of rows of a CTA that have
none, with and without the skip gradient."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [256, 512, 768, 1024, 1536, 2048, 3072, 4096, 5120, 6144, 8192])
@pytest.mark.parametrize("rows", [1, 2, 3, 15, 17, 149, 297, 593, 1187, 2371])
@pytest.mark.parametrize("rms,skip", [(False, True), (True, True), (False, False)])
def test_against_64_bits(D, rows, rms, skip):
    torch.manual_seed(rows + D)
    x, dy, add = ((torch.randn(rows, D, device="cuda") + 0.3).to(torch.bfloat16) for _ in range(3))
    g = torch.randn(D, device="cuda").to(torch.bfloat16)
    b = None if rms else torch.randn(D, device="cuda").to(torch.bfloat16)
    _, mean, rstd = native.norm_fwd(x, g, b, 1e-5, rms)
    dx, dg, db = native.norm_bwd(x, dy, g, mean, rstd, rms, dx_add=add if skip else None)
    xd, gd, bd = x.double().requires_grad_(), g.double().requires_grad_(), torch.zeros(D, dtype=torch.float64, device="cuda", requires_grad=True)
    mu = 0 if rms else xd.mean(-1, keepdim=True)
    y = (xd - mu) * ((xd - mu).square().mean(-1, keepdim=True) + 1e-5).rsqrt() * gd + bd
    y.backward(dy.double())
    want = xd.grad + (add.double() if skip else 0)
    # fp32 sums, one rounding to bf16: 2^-9 at most, 1.7e-3 in the mean
    assert (dx.double() - want).norm() <= 2.5e-3 * want.norm()
    assert (dg.double() - gd.grad).norm() <= 2.5e-3 * gd.grad.norm()
    assert rms or (db.double() - bd.grad).norm() <= 2.5e-3 * bd.grad.norm()
    assert _lib.read_status() == 0
