"""A transformer block as one native call each way against the same block operator by operator: the forward makes the same
launches, so the outputs are equal bit for bit; gradients agree to within what the order of fp32 additions in the attention
backward and in the bias gradients leaves (a last bit of bf16 here and there)."""
import copy

import pytest
import torch
import torch.utils.checkpoint

from ml_framework_b200 import _lib
from ml_framework_b200.engine import EngineConfig, TrainEngine
from ml_framework_b200.models.gpt import GPT, GPTConfig
from ml_framework_b200.models.llama import Llama, LlamaConfig
from ml_framework_b200.ops import block as block_mod
from ml_framework_b200.ops.block import whole_blocks
from ml_framework_b200.parallel.flat import FlatParams

pytestmark = pytest.mark.gpu


def _model(kind, layers=1):
    torch.manual_seed(3)
    if kind == "gpt":
        m = GPT(GPTConfig(layers, 256, 2, 1024, 500, 1024), torch.bfloat16, "cuda")
    else:
        m = Llama(LlamaConfig(layers, 512, 4, 2, 128, 1024, 500, 1024), torch.bfloat16, "cuda")
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
    return m


def _width(blk):
    return next(blk.parameters()).numel()          # the first normalisation's gamma


@pytest.fixture
def calls(monkeypatch):
    seen = []
    real = block_mod._BlockFn.apply
    monkeypatch.setattr(block_mod._BlockFn, "apply", lambda *a: (seen.append(1), real(*a))[1])
    return seen


def _pass(blk, x, dy, on):
    xin = x.clone().requires_grad_()
    h = xin * 1
    with whole_blocks(on):
        y = blk(h)
    y.backward(dy)
    return y.detach(), xin.grad


def _close(a, b):
    return (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()


@pytest.mark.parametrize("kind", ["gpt", "llama"])
@pytest.mark.parametrize("B,S", [(1, 1), (1, 37), (3, 129), (2, 256), (1, 600)])
@pytest.mark.parametrize("sink", [True, False])
def test_same_as_operators(kind, B, S, sink, calls):
    blk = _model(kind).blocks[0]
    other = copy.deepcopy(blk)
    ready = []
    if sink:
        for b in (blk, other):
            FlatParams(list(b.parameters()))
        for p in blk.parameters():
            p.grad_ready = ready.append
    x, dy = (torch.randn(B, S, _width(blk), device="cuda").to(torch.bfloat16) for _ in range(2))
    for step in range(2):                          # the second pass adds to the gradients of the first
        y, dx = _pass(blk, x, dy, True)
        y2, dx2 = _pass(other, x, dy, False)
        assert torch.equal(y, y2) and _close(dx, dx2)
        for (name, p), p2 in zip(blk.named_parameters(), other.parameters()):
            g, g2 = (p.main_grad, p2.main_grad) if sink else (p.grad, p2.grad)
            # one key: the softmax is 1 whatever the queries and keys are, and their gradients are rounding errors
            if S == 1 and "qkv" in name:
                g, g2 = g[-2 * 128:], g2[-2 * 128:]
            assert _close(g, g2), (name, step)
            assert not sink or p.grad is None
        if sink:
            assert len(ready) == (step + 1) * len(list(blk.parameters())) and {id(p) for p in ready} == {id(p) for p in blk.parameters()}
    assert len(calls) == 2 and _lib.read_status() == 0


@pytest.mark.parametrize("kind", ["gpt", "llama"])
def test_everything_else_runs_operator_by_operator(kind, calls):
    blk = _model(kind).blocks[0]
    d = _width(blk)
    x, dy = (torch.randn(2, 64, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    _pass(blk, x, dy, True)
    assert len(calls) == 1
    # off by default, and under no_grad
    _pass(blk, x, dy, False)
    with whole_blocks(), torch.no_grad():
        blk(x)
    # hooks on what is called inside
    fired = []
    for m in (blk.attn, blk.attn.qkv, blk.attn.proj, blk.mlp):
        h = m.register_forward_hook(lambda *a: fired.append(1) and None)
        _pass(blk, x, dy, True)
        h.remove()
    assert len(fired) == 4
    h = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    _pass(blk, x, dy, True)
    h.remove()
    # a frozen parameter, an input that needs no gradient, rows that are not packed, fp32 gradients
    blk.attn.qkv.weight.requires_grad_(False)
    _pass(blk, x, dy, True)
    blk.attn.qkv.weight.requires_grad_(True)
    with whole_blocks():
        blk(x).backward(dy)
    wide = torch.randn(2, 64, d + 8, device="cuda").to(torch.bfloat16).requires_grad_()
    assert block_mod.block(blk.ln1 if kind == "gpt" else blk.norm1, blk.attn, blk.ln2 if kind == "gpt" else blk.norm2, blk.mlp,
                           blk.mlp.fc1 if kind == "gpt" else blk.mlp.gate_up, blk.mlp.fc2 if kind == "gpt" else blk.mlp.down,
                           wide[..., :d], None, kind != "gpt") is None
    w = blk.attn.qkv.weight
    w.main_grad = torch.zeros(w.shape, device="cuda")
    _pass(blk, x, dy, True)
    assert w.main_grad.abs().sum() > 0
    del w.main_grad
    # a layer of another class
    class Other(type(blk.attn.proj)):
        pass
    blk.attn.proj.__class__ = Other
    _pass(blk, x, dy, True)
    assert len(calls) == 1


def test_saved_tensor_hooks_and_in_place_checks(calls):
    blk = _model("gpt").blocks[0]
    x, dy = (torch.randn(2, 96, 256, device="cuda").to(torch.bfloat16) for _ in range(2))
    want = _pass(blk, x, dy, True)
    with torch.autograd.graph.save_on_cpu():
        got = _pass(blk, x, dy, True)
    assert torch.equal(got[0], want[0]) and _close(got[1], want[1])
    xin = x.clone().requires_grad_()
    with whole_blocks():
        y = blk(xin * 1)
    with torch.no_grad():
        blk.mlp.fc2.weight.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(dy)
    assert len(calls) == 3


class _Recomputed(torch.nn.Module):
    def __init__(self, inner, reentrant):
        super().__init__()
        self.inner, self.reentrant = inner, reentrant

    def forward(self, x):
        return torch.utils.checkpoint.checkpoint(self.inner, x, use_reentrant=self.reentrant)


@pytest.mark.parametrize("kind", ["gpt", "llama"])
@pytest.mark.parametrize("how", ["torch", "torch reentrant", "package"])
def test_recomputed_blocks_under_the_engine(kind, how, calls):
    """What is recomputed in the backward takes the forward's path: torch's checkpoint compares the tensors that both save."""
    grads, losses = [], []
    ids, targets = (torch.randint(0, 500, (2, 128), device="cuda", generator=torch.Generator("cuda").manual_seed(n)) for n in (1, 2))
    for wrap in (False, True):
        m = _model(kind, layers=2)
        if wrap and how == "package":
            m.cfg.activation_checkpointing = True
        elif wrap:
            m.blocks = torch.nn.ModuleList(_Recomputed(b, how != "torch") for b in m.blocks)
        eng = TrainEngine(m, EngineConfig(strategy="none"))
        calls.clear()
        losses.append(eng.step(ids, targets).item())
        grads.append(eng.flat.grad.clone())
    # the loss is an fp32 sum over 256 rows in any order
    assert abs(losses[0] - losses[1]) <= 256 * 2.0 ** -24 * losses[0] and _close(grads[1], grads[0])
    # two blocks, in the forward where it records gradients (torch's own form) and where they are recomputed
    assert len(calls) == (4 if how == "torch" else 2)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("kind", ["gpt", "llama"])
def test_a_parameter_used_twice(kind, calls):
    """Its second gradient is added to the first."""
    blk = _model(kind).blocks[0]
    if kind == "gpt":
        blk.ln2.weight = blk.ln1.weight
    else:
        blk.norm2.weight = blk.norm1.weight
    other = copy.deepcopy(blk)
    x, dy = (torch.randn(2, 64, _width(blk), device="cuda").to(torch.bfloat16) for _ in range(2))
    for b, on in ((blk, True), (other, False)):
        FlatParams(list(b.parameters()))
        _pass(b, x, dy, on)
    for (name, p), p2 in zip(blk.named_parameters(), other.parameters()):
        assert _close(p.main_grad, p2.main_grad), name


@pytest.mark.parametrize("whole", [True, False])
@pytest.mark.parametrize("without", ["weight", "bias"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_normalisation_with_one_gradient_buffer(whole, without, dtype):
    """Gamma has a gradient buffer and beta none, or the other way round: each is written or added to by its own state."""
    blk = _model("gpt").blocks[0]
    p, q = (blk.ln1.bias, blk.ln1.weight) if without == "weight" else (blk.ln1.weight, blk.ln1.bias)
    p.main_grad, p._main_grad_started = torch.zeros(p.shape, dtype=dtype, device="cuda"), False
    other = copy.deepcopy(blk).double()
    for step in range(2):
        x, dy = (torch.randn(2, 64, 256, device="cuda").to(torch.bfloat16) for _ in range(2))
        _pass(blk, x, dy, whole)
        _pass(other, x.double(), dy.double(), False)
    p2, q2 = (other.ln1.bias, other.ln1.weight) if without == "weight" else (other.ln1.weight, other.ln1.bias)
    # bf16 activations in a chain of eight operators against none rounded
    for got, want in ((p.main_grad, p2.grad), (q.grad, q2.grad)):
        assert (got.double() - want).norm() <= 2e-2 * want.norm()
    assert p.grad is None
