"""Products with 129 - 511 rows, on CTA pairs or single CTAs: against the fp32 statement, around the row and column counts
where the route or the split of K changes."""
import pytest
import torch

from ml_framework_b200 import _lib as L
from ml_framework_b200.ops.gemm import gemm, gemm_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [128, 129, 255, 256, 257, 300, 511, 512])
@pytest.mark.parametrize("N,K", [(4096, 1024), (4112, 2056), (3136, 520), (3152, 1024), (12288, 512)])
@pytest.mark.parametrize("flags,b_mn", [(0, False), (0, True), (L.EPI_RESIDUAL, False), (L.EPI_SWIGLU, False), (L.EPI_ACCUM, False)])
def test_middle_rows(M, N, K, flags, b_mn):
    torch.manual_seed(M)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    b = w.t().contiguous() if b_mn else w
    aux = torch.randn(M, N, device="cuda").to(torch.bfloat16) if flags & L.EPI_RESIDUAL else None
    prev = torch.randn(M, N, device="cuda").to(torch.bfloat16) if flags & L.EPI_ACCUM else None
    want, _ = gemm_reference(a, b, b_mn=b_mn, aux_in=aux, flags=flags, prev_out=prev)
    got = gemm(a, b, b_mn=b_mn, aux_in=aux, flags=flags, out=prev)
    torch.cuda.synchronize()
    # one rounding to bf16; up to 256 rows and from 512 on a plain product may be the bf16 sum of up to eight partial
    # products: eight roundings of values below 8 (the largest of 2 M unit normals, 2^-6 each) at most
    split = (M <= 256 or M >= 512) and (flags & ~L.EPI_ACCUM) == 0
    tol = 8 * 2 ** -6 if split else 5e-4
    assert bool(((got.float() - want).abs() <= 2 ** -8 * want.abs() + tol).all())
    assert L.read_status() == 0
