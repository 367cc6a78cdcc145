"""Kernels launched with programmatic overlap: a chain of dependent launches gives what the operators give one by one,
at the sizes where the early weight loads end (runs shorter than the ring, remainders, each token-tile width)."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.ops import native
from ml_framework_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 32, 33, 64, 128, 129, 256])
@pytest.mark.parametrize("N,K", [(1024, 512), (1096, 2048), (4096, 5120)])
@pytest.mark.parametrize("shared", [False, True])
def test_chain_with_static_weights(M, N, K, shared):
    """norm -> product -> product -> norm ... with no ordinary launch in between. Every round has rows of its own, so that a
    read ahead of its time sees another round's values; with ``shared`` the rounds clear and fill one and the same buffer,
    so that a clear ahead of its time takes the round before's values from its second product."""
    torch.manual_seed(M + N)
    rounds = 6
    xs = [torch.randn(M, K, device="cuda").to(torch.bfloat16) for r in range(rounds)]
    g = torch.rand(K, device="cuda").to(torch.bfloat16)
    w1 = (torch.randn(N, K, device="cuda") * K ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(K, N, device="cuda") * N ** -0.5).to(torch.bfloat16)
    flags = _lib.EPI_ACCUM | _lib.EPI_B_STATIC
    mids = [torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(1 if shared else rounds)] * (rounds if shared else 1)
    ress = [x.clone() for x in xs]
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000)             # the host gets ahead: the launches stand back to back
    for x, mid, res in zip(xs, mids, ress):
        h, _, _ = native.norm_fwd(x, g, None, 1e-5, True, want_stats=False, zero=mid)
        gemm(h, w1, out=mid, flags=flags)
        gemm(mid, w2, out=res, flags=flags)
    torch.cuda.synchronize()
    rms = lambda t: t.pow(2).mean().sqrt().item()
    for r, (x, mid, res) in enumerate(zip(xs, mids, ress)):
        xf = x.float()
        hf = (xf * torch.rsqrt((xf * xf).mean(-1, keepdim=True) + 1e-5) * g.float()).to(torch.bfloat16).float()
        mf = hf @ w1.float().t()
        # every partial tile is added in bf16: at most one rounding (2^-9 of the running value) per SM that shares the tile,
        # and a value at a rounding boundary of h may round the other way; 4 sigma of that in the root mean square
        if not shared or r == rounds - 1:
            assert rms(mid.float() - mf) <= 2 ** -7 * rms(mf), r
        # the same for the second product, whose rows (unit norm) carry the first one's error on
        rf = xf + mf @ w2.float().t()
        assert rms(res.float() - rf) <= 2 ** -7 * (rms(rf) + rms(mf)), r
    assert _lib.read_status() == 0


@pytest.mark.parametrize("rows,D", [(1, 256), (5, 1024), (3, 2048), (300, 4096), (2, 5120)])
@pytest.mark.parametrize("zero_elems", [8, 16384 + 8, 5_000_000])
def test_norm_clears_a_buffer(rows, D, zero_elems):
    torch.manual_seed(0)
    x = torch.randn(rows, D, device="cuda").to(torch.bfloat16)
    g = torch.rand(D, device="cuda").to(torch.bfloat16)
    guard = torch.ones(zero_elems + 64, device="cuda", dtype=torch.bfloat16)
    y0, _, _ = native.norm_fwd(x, g, None, 1e-5, True, want_stats=False)
    y1, _, _ = native.norm_fwd(x, g, None, 1e-5, True, want_stats=False, zero=guard[:zero_elems])
    assert torch.equal(y0, y1)
    assert not guard[:zero_elems].any() and bool((guard[zero_elems:] == 1).all())
    assert _lib.read_status() == 0


@pytest.mark.parametrize("M,flags", [(256, 0), (256, _lib.EPI_B_STATIC), (512, 0)])
def test_wait_budget_starts_behind_the_kernels_ahead(M, flags):
    """A pair product becomes resident beside a long decode kernel of one CTA (some 0.9 ms for 64 Ki tokens): the time until
    that kernel's end is not part of the product's own wait budget (400,000 cycles, 0.2 ms; its waits are microseconds)."""
    from ml_framework_b200.dist.symm import set_wait_budget_cycles
    torch.manual_seed(M)
    n, bs = 65536, 16
    cache = torch.randn(n // bs, 2, bs, 1, 128, device="cuda").to(torch.bfloat16)
    table = torch.arange(n // bs, dtype=torch.int32, device="cuda")[None]
    lens = torch.tensor([n], dtype=torch.int32, device="cuda")
    q = torch.randn(1, 1, 128, device="cuda").to(torch.bfloat16)
    a = torch.randn(M, 2048, device="cuda").to(torch.bfloat16)
    w = (torch.randn(4096, 2048, device="cuda") * 2048 ** -0.5).to(torch.bfloat16)
    bias = torch.randn(4096, device="cuda").to(torch.bfloat16)
    want = (a.double() @ w.double().t() + bias.double()).float()
    out = torch.zeros(M, 4096, device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    set_wait_budget_cycles(400_000)
    try:
        native.paged_decode(q, cache, table, lens, n, split_tokens=n)
        gemm(a, w, out=out, bias=bias, flags=flags)
        status = _lib.read_status()
    finally:
        set_wait_budget_cycles(0)
    assert status == 0
    # one rounding to bf16 and the fp32 sum of 2048 products of order 2^-5
    assert bool(((out.float() - want).abs() <= 2 ** -8 * want.abs() + 5e-4).all())
