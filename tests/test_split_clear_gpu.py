"""A product whose K is split clears its output first: its own columns and no others, whole vectors or not."""
import pytest
import torch

from ml_framework_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1024, 1000, 8192), (520, 257, 4096), (513, 263, 4096)])
def test_clears_its_columns_only(M, N, K):
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    buf = torch.full((M, 1024 + 8), 1000.0, dtype=torch.bfloat16, device="cuda")
    gemm(a, b, out=buf[:, :N])
    want = a.double() @ b.double().T
    # partial sums of up to 8 splits meet in bf16
    assert ((buf[:, :N].double() - want).abs() <= 9 * 2.0 ** -9 * (want.abs() + 6 * K ** 0.5)).all()
    assert (buf[:, N:] == 1000).all()
