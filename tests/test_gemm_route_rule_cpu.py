"""Which kernel takes a product of more than a few rows: CTA pairs or single CTAs."""
import pytest

from ml_framework_b200 import _lib

ACC, F32, RES, STATIC = _lib.EPI_ACCUM, _lib.EPI_OUT_FP32, _lib.EPI_RESIDUAL, _lib.EPI_B_STATIC


@pytest.mark.parametrize("M,N,K,flags,comm,pairs", [
    (128, 8192, 4096, 0, 0, 0), (129, 8192, 4096, 0, 0, 1), (512, 2048, 256, 0, 0, 1), (512, 1792, 256, 0, 0, 0), (8192, 768, 768, ACC, 0, 1),
    # 129 - 511 rows: single CTAs while their 128 x 64 tiles run at once, pairs from the next tile column on
    (129, 4032, 512, RES, 0, 0), (256, 4095, 512, RES, 0, 0), (256, 4096, 512, RES, 0, 1),
    (300, 2048, 8192, 0, 0, 0), (300, 3136, 3072, STATIC, 0, 0), (300, 3137, 3072, 0, 0, 1), (400, 2368, 2304, 0, 0, 0), (400, 2369, 2304, 0, 0, 1),
    (300, 2048, 4096, _lib.EPI_DSWIGLU, 0, 1), (300, 2048, 4104, _lib.EPI_DSWIGLU, 0, 0),
    (300, 3072, 1024, _lib.EPI_GELU | _lib.EPI_STORE_PRE, 0, 1), (300, 3072, 1024, _lib.EPI_GELU, 0, 0),
    (257, 4096, 1024, 0, 0, 1), (511, 28672, 4096, 0, 0, 1),
    # rounds: 1.8 against 1, then 2 against 2; 5.8 against 4
    (300, 12288, 4096, 0, 0, 0), (300, 12288, 4096, _lib.EPI_GELU, 0, 1), (385, 12288, 4096, 0, 0, 1), (300, 50304, 2048, 0, 0, 1),
    # fp32 outputs
    (300, 50304, 2048, F32, 0, 0), (300, 18944, 2048, F32, 0, 1), (300, 6144, 1024, F32, 0, 0), (300, 4096, 1024, F32, 0, 1), (300, 6144, 2048, F32, 0, 1),
    # an accumulation keeps its fp32 addition, rows that travel their fixed line
    (511, 8192, 4096, ACC, 0, 0), (511, 8192, 4096, 0, 1, 0), (512, 8192, 4096, 0, 1, 1)])
def test_route_on_148_sms(M, N, K, flags, comm, pairs):
    assert _lib.get().mlf_gemm_takes_pairs(M, N, K, flags, comm, 148) == pairs


def test_every_shape_has_an_answer():
    f = _lib.get().mlf_gemm_takes_pairs
    for sms in (148, 132, 2, 1):
        for M in (1, 128, 129, 256, 257, 384, 385, 511, 512):
            for N in (8, 511, 512, 2048, 4095, 4096, 12288, 50304):
                assert f(M, N, 1024, 0, 0, sms) in (0, 1)
