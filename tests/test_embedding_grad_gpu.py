"""Embedding gradient summed per token's row instead of in an fp32 table, against 64-bit sums: few and many repeats, ids outside the
table, more tokens than rows."""
import pytest
import torch

from ml_framework_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,V,D", [(1, 50, 8), (49, 50, 264), (50, 50, 264), (513, 50, 1024), (513, 5000, 1024), (2331, 50304, 256)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("spread", ["all", "few", "one"])
def test_against_64_bit_sums(T, V, D, accumulate, spread):
    torch.manual_seed(T)
    native.embedding_grad(torch.randn(T, D, device="cuda").to(torch.bfloat16), torch.randint(0, V, (T,), device="cuda"),
                          torch.empty(V, D, dtype=torch.bfloat16, device="cuda"))      # leaves other ids' owners in the scratch
    ids = torch.randint(0, {"all": V, "few": min(V, 7), "one": 1}[spread], (T,), device="cuda")
    if T > 1:
        ids[0], ids[-1] = V + 3, -1                   # outside the table: skipped
    dout = torch.randn(T, D, device="cuda").to(torch.bfloat16)
    out = torch.randn(V, D, device="cuda").to(torch.bfloat16)
    start = out.double() if accumulate else torch.zeros(V, D, device="cuda", dtype=torch.float64)
    native.embedding_grad(dout, ids, out, accumulate)
    ok = (ids >= 0) & (ids < V)
    want = start.index_add(0, ids[ok], dout[ok].double())
    size = start.abs().index_add(0, ids[ok], dout[ok].double().abs())
    # an fp32 sum of T terms in any order, and one rounding to bf16
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + T * 2.0 ** -24 * size).all()
