"""Copies that a wrapper makes of its arguments (packed rows, packed ids) live until the kernel is queued: freed earlier, their
memory could be given to the next copy."""
import weakref

import pytest
import torch

from ml_framework_b200.ops import native

BF = torch.bfloat16


def _wide(*shape, dtype=BF):
    """A tensor of this shape whose rows are not packed."""
    return torch.ones(*shape[:-1], 2 * shape[-1], dtype=dtype)[..., ::2] if len(shape) == 1 else torch.ones(*shape[:-1], shape[-1] + 1, dtype=dtype)[..., :-1]


def _ids(*shape):
    return _wide(*shape, dtype=torch.int64)


CALLS = {
    "gelu_bwd": lambda: native.gelu_bwd(_wide(4, 8), _wide(4, 8)),
    "swiglu_bwd": lambda: native.swiglu_bwd(_wide(4, 8), torch.ones(4, 16, dtype=BF)),
    "embedding_fwd": lambda: native.embedding_fwd(_ids(2, 4), torch.ones(9, 8, dtype=BF), torch.arange(4).expand(2, 4), torch.ones(4, 8, dtype=BF)),
    "embedding_bwd": lambda: native.embedding_bwd(_wide(2, 4, 8), _ids(2, 4), 9),
    "embedding_grad": lambda: native.embedding_grad(_wide(2, 4, 8), _ids(2, 4), torch.ones(9, 8, dtype=BF)),
    "rope_": lambda: native.rope_(torch.ones(4, 2, 8, dtype=BF), _ids(4), 1e4),
    "rope_qkv": lambda: native.rope_qkv(torch.ones(4, 3 * 128, dtype=BF), _ids(4), 1, 1, 1e4),
    "cross_entropy_": lambda: native.cross_entropy_(torch.ones(4, 16, dtype=BF), _ids(4), 9),
    "paged_decode_rope": lambda: native.paged_decode_rope(
        torch.ones(4, 3 * 128, dtype=BF), torch.ones(8, 2, 16, 1, 128, dtype=BF), torch.zeros(4, 2, dtype=torch.int32), _wide(4, dtype=torch.int32),
        _ids(4), 1, 1, 32, 1e4, split_tokens=128),
    "kv_cache_write": lambda: native.kv_cache_write(torch.ones(8, 2, 16, 1, 128, dtype=BF), *(torch.ones(4, 1, 128, dtype=BF),) * 2, _ids(4)),
    "rope_kv_write_": lambda: native.rope_kv_write_(torch.ones(4, 3 * 128, dtype=BF), _ids(4), _ids(4), torch.ones(8, 2, 16, 1, 128, dtype=BF), 1, 1, 1e4),
}


@pytest.mark.parametrize("name", CALLS)
def test_copies_live_until_the_launch(name, monkeypatch):
    taken, launches = [], []

    class Function:
        def __init__(self, fn):
            self.fn = fn

        def __call__(self, *args):
            if self.fn.endswith(("_bytes", "_elems")):
                return 1024
            launches.append([ref() is not None for ref in taken])
            return 0

    class Library:
        def __getattr__(self, fn):
            return Function(fn)

    real = native._p
    monkeypatch.setattr(native, "_p", lambda t: (taken.append(weakref.ref(t)) if t is not None else None, real(t))[1])
    monkeypatch.setattr(native, "_L", Library)
    monkeypatch.setattr(native, "_st", lambda: 0)
    CALLS[name]()
    assert len(launches) == 1 and launches[0] and all(launches[0])
