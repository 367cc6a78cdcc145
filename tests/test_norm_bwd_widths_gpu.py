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


@pytest.mark.parametrize("D", [256, 512, 768, 1024, 1536, 2048, 3072, 4096, 5120, 6144, 8192])
def test_rows_far_from_zero(D):
    """x - mean is formed before it is scaled: rows of 1000 +- 4 keep the digits that x * rstd - mean * rstd would round away."""
    torch.manual_seed(D)
    x = 1000 + 4 * (torch.randint(0, 2, (2, D), device="cuda") * 2 - 1).to(torch.bfloat16)
    dy = torch.randn(2, D, device="cuda").to(torch.bfloat16)
    g = torch.ones(D, device="cuda").to(torch.bfloat16)
    mean = torch.full((2,), 1000.0, device="cuda")
    rstd = torch.tensor([0.24999992, 0.2371823], device="cuda")
    dg, db = (torch.empty(D, device="cuda") for _ in range(2))
    native.norm_bwd(x, dy, g, mean, rstd, False, dgamma_out=dg, dbeta_out=db)
    terms = dy.double() * (x.double() - 1000) * rstd.double()[:, None]
    # two products and a sum per row, and the sum of both rows, in fp32
    assert ((dg.double() - terms.sum(0)).abs() <= 8 * 2.0 ** -24 * terms.abs().sum(0)).all()
