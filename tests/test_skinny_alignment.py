"""Rows of the weight-streaming products are read by 16 bytes: what does not start there is copied or refused, never launched (no GPU needed)."""
import pytest
import torch

from cisr_b200.ops import build, kernels


def off_by(n, *shape):
    """A contiguous bfloat16 tensor that starts n elements behind a 16-byte boundary."""
    flat = torch.zeros(shape[0] * shape[1] + 16, dtype=torch.bfloat16)
    start = -flat.data_ptr() // 2 % 8 + n
    return flat[start:start + shape[0] * shape[1]].view(*shape)


@pytest.mark.parametrize("field", [0, 1, 2, 3, 5])       # w, act, x, delta, x_out
def test_entry_refuses_misaligned_rows(field):
    addresses = [1 << 40] * 19
    addresses[field] += 2
    assert build.load_library("skinny_gemm.cu").cisr_skinny_gemm(kernels._SKINNY_CALL.pack(*addresses, 1e-5, 1.0, 0.0, 64, 64, 0, 4, 0, 0, *[0] * 9)) == -2


def test_feed_forward_copies_activations_that_start_off_a_boundary(monkeypatch):
    seen = []

    class Library:
        def cisr_skinny_chain(self, args, n):
            seen.append(kernels._SKINNY_PAIR.unpack(args)[1])
            return 0

    monkeypatch.setattr(kernels, "_need", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "_skinny", Library)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    gate_up, down = off_by(0, 32, 16), off_by(0, 8, 16)
    for n in (0, 1, 4):
        h = off_by(n, 4, 16)
        kernels.skinny_mlp(h, gate_up, down)
        assert seen[-1] % 16 == 0 and (n or seen[-1] == h.data_ptr())
