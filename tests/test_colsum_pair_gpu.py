"""Column sums of two matrices in one launch: widths that end inside a column block, few and many rows, added or written."""
import ctypes as C

import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 33, 2331])
@pytest.mark.parametrize("N0,N1", [(256, 768), (1024, 4096), (8, 264), (300, 20)])
@pytest.mark.parametrize("acc0,acc1", [(0, 0), (1, 0), (0, 1)])
def test_pair_against_64_bit_sums(M, N0, N1, acc0, acc1):
    torch.manual_seed(M + N0)
    dy = [torch.randn(M, (n + 7) // 8 * 8 + 8, device="cuda").to(torch.bfloat16) for n in (N0, N1)]
    db = [torch.randn(n + 8, device="cuda").to(torch.bfloat16) for n in (N0, N1)]
    was = [t.clone() for t in db]
    sc = native.colsum_scratch(M, ((N0, N1),), torch.device("cuda", 0))
    args = [x for t, d, n, a in zip(db, dy, (N0, N1), (acc0, acc1))
            for x in (C.c_void_p(t.data_ptr()), C.c_void_p(d.data_ptr()), n, C.c_longlong(d.stride(0)), a)]
    for _ in range(2):                                     # the counters are zero again after the first
        for t, w in zip(db, was):
            t.copy_(w)
        _lib.check(_lib.get().mlf_colsum2(*args, M, C.c_void_p(sc.data_ptr()), C.c_uint64(_lib.stream_handle())), "mlf_colsum2")
    for t, w, d, n, a in zip(db, was, dy, (N0, N1), (acc0, acc1)):
        terms = d[:, :n].double()
        want = terms.sum(0) + a * w[:n].double()
        # an fp32 sum of M + 1 terms, one rounding to bf16
        bound = 2.0 ** -8 * want.abs() + (M + 1) * 2.0 ** -24 * (terms.abs().sum(0) + w[:n].double().abs())
        assert ((t[:n].double() - want).abs() <= bound).all()
        assert torch.equal(t[n:], w[n:])
