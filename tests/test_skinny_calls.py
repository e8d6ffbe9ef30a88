"""What the weight-streaming products are handed: rows, read by 16 bytes, that do not start there; rotations without tables (no GPU needed)."""
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


def test_rotation_without_tables_or_pairing(monkeypatch):
    """A head without rotation needs neither tables nor the order of its pairs."""
    seen = []

    class Library:
        def cisr_skinny_gemm(self, args):
            seen.append(kernels._SKINNY_CALL.unpack(args))
            return 0

    monkeypatch.setattr(kernels, "_need", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "_skinny", Library)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    ints, cache = torch.zeros(2, 3, dtype=torch.int32), off_by(0, 4, 32)
    rope = dict(rot_half=0, q_out=cache, k_cache=cache, v_cache=cache, positions=ints, token_req=ints, req_slot=ints, block_table=ints, page_size=2, hq=1, hkv=1, dim=16)
    kernels.skinny_gemm(off_by(0, 48, 32), 2, act=off_by(0, 2, 32), epilogue=kernels.EPI_ROPE, rope=rope)
    assert seen[0][9:11] == (0, 0) and seen[0][28:30] == (0, 0)      # cos, sin; rot_half, interleaved
