"""CTA-pair GEMM whose last round of tiles is cut into items of 128 columns: every epilogue and
operand layout, ragged last tiles, fewer tiles than half a round."""
import pytest
import torch

from ml_framework_b200 import _lib as L
from ml_framework_b200.ops.gemm import gemm, gemm_reference

pytestmark = pytest.mark.gpu

KINDS = {"plain": 0, "gelu_pre": L.EPI_GELU | L.EPI_STORE_PRE, "residual": L.EPI_RESIDUAL, "dgelu": L.EPI_DGELU_MUL, "swiglu": L.EPI_SWIGLU,
         "dswiglu": L.EPI_DSWIGLU, "fp32": L.EPI_OUT_FP32}
# 256 x 256 tiles: 76 and 78 (a round of 74 and a few), 16 (less than half a round), 257 (three rounds and half of one)
SHAPES = [(4864, 1024, 320), (3300, 1424, 1096), (1024, 1008, 512), (512, 2048, 1152), (65700, 256, 192)]


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_half_width_items(kind, M, N, K):
    torch.manual_seed(M + K)
    flags = KINDS[kind]
    r = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    a, b = r(M, K), (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    bias = r(N) if kind in ("plain", "gelu_pre", "residual") else None
    aux = r(M, 2 * N if flags & L.EPI_DSWIGLU else N) if flags & (L.EPI_RESIDUAL | L.EPI_DGELU_MUL | L.EPI_DSWIGLU) else None
    pre = torch.full((M, N), 9.0, device="cuda", dtype=torch.bfloat16) if flags & L.EPI_STORE_PRE else None
    want, want_pre = gemm_reference(a, b, bias=bias, aux_in=aux, flags=flags | (L.EPI_BIAS if bias is not None else 0))
    guard = torch.full((M + 8, want.shape[1]), 5.0, device="cuda", dtype=torch.float32 if kind == "fp32" else torch.bfloat16)
    got = gemm(a, b, out=guard[:M], bias=bias, aux_in=aux, aux_out=pre, flags=flags, out_dtype=guard.dtype)
    torch.cuda.synchronize()
    # one rounding to bf16 (2^-8 of the value at most) and the fp32 product and activation, whose error is below 1e-4 of
    # the operands' order of magnitude (1)
    ok = lambda x, y: bool(((x.float() - y).abs() <= 2 ** -8 * y.abs() + 5e-4).all())
    assert ok(got, want)
    if pre is not None:
        assert ok(pre, want_pre)
    assert bool((guard[M:] == 5.0).all())
    assert L.read_status() == 0


@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(4864, 1024, 320), (3304, 1424, 1096), (512, 2048, 960)])
def test_half_width_items_layouts(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + K)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    got = gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    want = a.float() @ b.float().t()
    # as above; K is too short, or the rounds too many, for partial sums that meet in bf16
    assert bool(((got.float() - want).abs() <= 2 ** -8 * want.abs() + 5e-4).all())
    assert L.read_status() == 0
