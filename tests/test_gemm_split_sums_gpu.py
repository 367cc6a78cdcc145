"""Products that split K into few parts or not at all (99 - 116 tiles, 129 - 256 rows): error against 64 bits."""
import pytest
import torch

from ml_framework_b200 import _lib as L
from ml_framework_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1280, 5120, 8192), (2560, 2560, 2560), (2048, 3328, 4096), (2048, 3584, 8192), (1024, 7168, 4096), (256, 28672, 4096)])
def test_no_more_than_two_partial_sums(M, N, K):
    torch.manual_seed(M)
    a, b = torch.randn(K, M, device="cuda").to(torch.bfloat16), (torch.randn(K, N, device="cuda") * K ** -0.5).to(torch.bfloat16)
    want = a.double().t() @ b.double()
    two = (a[:K // 2].float().t() @ b[:K // 2].float()).to(torch.bfloat16) + (a[K // 2:].float().t() @ b[K // 2:].float()).to(torch.bfloat16)
    rel = lambda x: float((x.double() - want).norm() / want.norm())
    got = gemm(a, b, a_mn=True, b_mn=True)
    # two partial sums, each rounded to bf16 and added in bf16; over millions of elements the error of the same number of
    # roundings repeats to well below a tenth, and three partial sums have 1.16 times that of two
    assert rel(got) <= 1.05 * rel(two)
    assert L.read_status() == 0


@pytest.mark.parametrize("M,N,K,switch", [(200, 4096, 1000, 1), (129, 6144, 1016, 1), (256, 4096, 968, 1), (200, 4096, 4096, 0), (256, 6144, 2048, 0), (200, 2048, 2048, 0)])
def test_one_fp32_sum(M, N, K, switch):
    """K just short of the small-M split's line, and the split switched off: a single rounding to bf16."""
    torch.manual_seed(K)
    a, w = torch.randn(M, K, device="cuda").to(torch.bfloat16), (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    want = (a.double() @ w.double().t()).float()
    L.get().mlf_set_gemm_small_m_split(switch)
    try:
        got = gemm(a, w)
        torch.cuda.synchronize()
    finally:
        L.get().mlf_set_gemm_small_m_split(1)
    # half a unit in the last place of bf16 and the fp32 sum of K products of order K^-1/2
    assert bool(((got.float() - want).abs() <= 2 ** -8 * want.abs() + 5e-4).all())
    assert L.read_status() == 0
