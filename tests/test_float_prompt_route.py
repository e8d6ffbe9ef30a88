"""Which kernel float prompts take by where their buffers start: the tensor-core one reads rows by 16 bytes (no GPU needed)."""
import pytest
import torch

from cisr_b200.ops import build, kernels


def off_by(n, *shape):
    """A contiguous float tensor that starts n elements behind a 16-byte boundary."""
    size = torch.Size(shape).numel()
    flat = torch.zeros(size + 8)
    start = -flat.data_ptr() // 4 % 4 + n
    return flat[start:start + size].view(*shape)


@pytest.mark.parametrize("off", [(0, 0, 0), (1, 0, 0), (0, 2, 0), (0, 0, 3)])        # of q, k_cache, v_cache
def test_route(off, monkeypatch):
    taken = []

    class Library:
        def __init__(self, name):
            self.cisr_attn_prefill = self.cisr_attn_prefill_float = lambda *a: taken.append(name) or 0

    monkeypatch.setattr(kernels, "_need", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "_attention_float", lambda dim, softcap=False: Library("tensor cores"))
    monkeypatch.setattr(kernels, "attention_library", lambda dim, dtype, kind="auto", softcap=False: Library("multiply-adds"))
    q, k, v = off_by(off[0], 5, 2, 16), off_by(off[1], 3, 1, 16, 16), off_by(off[2], 3, 1, 16, 16)
    ints = torch.zeros(3, dtype=torch.int32)
    kernels.attn_prefill(q, off_by(1, 5, 2, 16), k, v, ints, ints[None], ints, ints, ints, ints, ints, 2, 1, 16, 0.25, None)
    assert taken == ["multiply-adds" if any(off) else "tensor cores"]


@pytest.mark.parametrize("field", [0, 2, 3])
def test_entry_refuses_what_it_cannot_read(field):
    at = [1 << 40] * 4
    at[field] += 4
    lib = build.load_library("attention_float.cu", {"HEAD_DIM": 16})
    assert lib.cisr_attn_prefill_float(*at, 0, 0, 1, 0, 0, 1, 0, 0, 0, 2, 1, 16, 0.25, 0.0, 0, 0, 0.0, 0, 0) == -2
