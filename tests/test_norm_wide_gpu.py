"""Normalisation forward at the widths that take one thread per vector of a row, or one warp per row when rows are many:
row counts around the change of the rows per CTA (twice two CTAs per SM), around the end of the grid and on both sides of
the change of the kernel."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native
from ml_framework_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [3072, 5120, 6144, 8192])
@pytest.mark.parametrize("rows", [1, 24, 297, 591, 593, 1185])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_fwd_one_vector_per_thread(rows, D, rms):
    _check(rows, D, rms)


@pytest.mark.parametrize("D,line", [(3072, 1184), (5120, 800), (6144, 800), (8192, 2304)])
@pytest.mark.parametrize("past", [-1, 0, 9500])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_fwd_one_warp_per_row(D, line, past, rms):
    _check(line + past, D, rms)


def _check(rows, D, rms):
    torch.manual_seed(rows)
    x = (torch.randn(rows, D, device="cuda") * 1.5 + 0.3).to(torch.bfloat16)
    g = (1 + 0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16)
    b = None if rms else (0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16)
    y, mean, rstd = native.norm_fwd(x, g, b, 1e-5, rms)
    if rms:
        yr, rr = ref.rms_norm_ref(x.float(), g.float(), 1e-5)
    else:
        yr, mr, rr = ref.layer_norm_ref(x.float(), g.float(), b.float(), 1e-5)
        assert (mean - mr.reshape(-1)).abs().max().item() < 1e-5      # fp32 sums of 3072 - 8192 values of order 1
    assert ((rstd - rr.reshape(-1)).abs() <= 1e-5 * rr.reshape(-1)).all()
    # one rounding to bf16 (half a unit in the last place: 2^-8 of the value at a power of two), and the fp32
    # statistics' own error
    assert ((y.float() - yr).abs() <= 2 ** -8 * yr.abs() + 1e-4).all()
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
