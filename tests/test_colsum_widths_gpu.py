"""Column sums of different widths share one scratch buffer per device: the counters of a wide matrix must still be zero after
narrower ones have left their partial sums in it."""
import torch
import pytest

from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [16384, 16640, 20480, 28672])
def test_wide_after_narrow(wide):
    torch.manual_seed(wide)
    x = torch.randn(300, wide, device="cuda").to(torch.bfloat16)
    native.colsum(x)                                    # the scratch has its size now
    for _ in range(2):
        for n in (256, 1024, 5120):
            native.colsum(x[:, :n])
        got = native.colsum(x)
        want = x.double().sum(0)
        # sums in fp32, one rounding to bf16
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()


@pytest.mark.parametrize("wide", [(1 << 19) + 264, (1 << 20) + 8])
def test_more_columns_than_counters(wide):
    torch.manual_seed(wide)
    x = torch.randn(40, wide, device="cuda").to(torch.bfloat16)
    want = x.double().sum(0)
    for _ in range(2):
        native.colsum(x[:, :256])
        got = native.colsum(x, out=torch.full_like(x[0], float("nan")))
        # sums in fp32, one rounding to bf16
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
