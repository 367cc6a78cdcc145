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
