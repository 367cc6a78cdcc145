"""Epilogues of the CTA-pair GEMM at ragged shapes: last tiles that reach into one half of the columns only, row tails,
several tiles per CTA pair, one and two epilogue warps per accumulator quarter (short and long K)."""
import pytest
import torch

from ml_framework_b200 import _lib as L
from ml_framework_b200.ops.gemm import gemm, gemm_reference

pytestmark = pytest.mark.gpu

KINDS = {"plain": 0, "gelu_pre": L.EPI_GELU | L.EPI_STORE_PRE, "residual": L.EPI_RESIDUAL, "dgelu": L.EPI_DGELU_MUL, "swiglu": L.EPI_SWIGLU,
         "swiglu_pre": L.EPI_SWIGLU | L.EPI_STORE_PRE, "dswiglu": L.EPI_DSWIGLU}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("M,N,K", [(1000, 1040, 64), (777, 2128, 1096), (2560, 2224, 192), (5000, 1200, 1160), (512, 8192, 2048)])
def test_ragged_epilogues(kind, M, N, K):
    torch.manual_seed(M + K)
    flags = KINDS[kind]
    r = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    a, b = r(M, K), (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    bias = r(N) if kind in ("plain", "gelu_pre", "residual") else None
    aux = r(M, 2 * N if flags & L.EPI_DSWIGLU else N) if flags & (L.EPI_RESIDUAL | L.EPI_DGELU_MUL | L.EPI_DSWIGLU) else None
    pre = torch.full((M, N), 9.0, device="cuda", dtype=torch.bfloat16) if flags & L.EPI_STORE_PRE else None
    want, want_pre = gemm_reference(a, b, bias=bias, aux_in=aux, flags=flags | (L.EPI_BIAS if bias is not None else 0))
    guard = torch.full((M + 8, want.shape[1]), 5.0, device="cuda", dtype=torch.bfloat16)
    got = gemm(a, b, out=guard[:M], bias=bias, aux_in=aux, aux_out=pre, flags=flags)
    torch.cuda.synchronize()
    # one rounding to bf16 (2^-8 of the value at most) and the fp32 product and activation, whose error is below 1e-4 of
    # the operands' order of magnitude (1)
    ok = lambda x, y: bool(((x.float() - y).abs() <= 2 ** -8 * y.abs() + 5e-4).all())
    assert ok(got, want)
    if pre is not None:
        assert ok(pre, want_pre)
    assert bool((guard[M:] == 5.0).all())
    assert L.read_status() == 0
