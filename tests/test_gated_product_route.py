"""From how many tokens on a gated product is one launch of the tcgen05 kernel, and what it gives there."""
import pytest
import torch

from cisr_b200.ops import kernels
from cisr_b200.parts import feedforward


def test_rule():
    def ok(tokens, rows, k, dtype=torch.bfloat16):
        return kernels.tcgen05_gated_ok(torch.empty(tokens, k, dtype=dtype), torch.empty(rows, k, dtype=dtype))
    assert not ok(16, 3072, 576) and ok(17, 3072, 576) and ok(127, 3072, 576)
    assert not ok(31, 16384, 2048) and ok(32, 16384, 2048)
    assert not ok(127, 28672, 4096) and ok(128, 28672, 4096)
    # 16 MB of weights and more: fewer than 128 KB of activations are the library's, which is ahead there by up to 1 us
    assert not ok(63, 8192, 1024) and ok(64, 8192, 1024) and not ok(42, 12288, 1536) and ok(43, 12288, 1536)
    assert not ok(64, 3072, 576, torch.float32) and not ok(64, 3072, 572)


@pytest.mark.gpu
@pytest.mark.parametrize("gate,limit", [("silu", None), ("gelu_tanh", None), ("gated_clamp", 1.5)])
@pytest.mark.parametrize("inter,k", [(1536, 576), (100, 64), (4000, 1024)])
def test_values(gate, limit, inter, k):
    g = torch.Generator().manual_seed(inter)
    w = (torch.randn(2 * inter, k, generator=g) * k ** -0.5).bfloat16().cuda()
    for tokens in (17, 31, 32, 33, 127):
        a = torch.randn(tokens, k, generator=g).bfloat16().cuda()
        assert kernels.tcgen05_gated_ok(a, w)
        want = torch.empty(tokens, inter, dtype=torch.bfloat16, device="cuda")
        kernels.swiglu(kernels.gemm_library(a, w, torch.empty(tokens, 2 * inter, device="cuda")), want, gate=gate, limit=limit)
        got = feedforward.gated_product(a, w, gate, limit)
        # the same float sums up to their order, then one rounding to bfloat16: at most a step apart
        torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -7, atol=1e-5)
    kernels.raise_if_kernel_gave_up()
