"""Serving a model whose head has no aligned number of rows."""
import pytest
import torch

from ml_framework_b200 import _lib
from ml_framework_b200.models.llama import Llama, LlamaConfig
from ml_framework_b200.serving.executor import ExecutorConfig, PagedLlamaExecutor
from ml_framework_b200.serving.kv_cache import KVCacheBlockManager
from ml_framework_b200.serving.scheduler import Batch, Request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [1000, 1001, 1004])
def test_unpadded_vocabulary(vocab):
    torch.manual_seed(0)
    cfg = LlamaConfig(n_layers=2, d_model=256, n_heads=2, n_kv_heads=1, head_dim=128, d_ff=512, vocab_size=vocab, max_seq=256, vocab_multiple=1)
    model = Llama(cfg, torch.bfloat16, "cuda").eval()
    with torch.no_grad():
        # a clear winner for every token, so that the two arms' roundings do not decide
        model.embed.weight.normal_(0, 1.0)
        model.lm_head.copy_(model.embed.weight.roll(1, 0) * 0.1)
    out = {}
    for torch_ops in (True, False):
        kv = KVCacheBlockManager(64, 16, cfg.head_dim, cfg.n_layers, cfg.n_kv_heads, device="cuda", dtype=torch.bfloat16)
        ex = PagedLlamaExecutor(model, kv, ExecutorConfig(max_batch=4, max_seq_len=256, prefill_chunk=64, torch_ops=torch_ops, graph_warmup_steps=1))
        reqs = [Request([(7 * i + 3 * j) % (vocab - 1) + 1 for j in range(9 + 4 * i)], max_tokens=6) for i in range(3)]
        for step in range(5):
            new = ex.execute_batch(Batch(reqs, **{"prefill" if step == 0 else "decode": reqs})).generated_tokens
            for r in reqs:
                r.generated.append(new[r.id])
        out[torch_ops] = [r.generated for r in reqs]
    assert all(len(t) == 5 for t in out[True]) and out[True] == out[False]
    assert _lib.read_status() == 0
