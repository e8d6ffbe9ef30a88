"""Which path a step's routed experts take, by sizes (no GPU needed)."""
import pytest
import torch


@pytest.mark.parametrize("experts,top,width,ff,gated,tokens,grouped", [
    (16, 4, 1024, 384, True, 32, False), (16, 4, 1024, 384, True, 64, True),              # a few small experts: three more launches have to pay
    (64, 8, 4096, 896, True, 4, False), (64, 8, 4096, 896, True, 16, True), (64, 8, 4096, 896, False, 8, False), (64, 8, 4096, 896, False, 24, True),
    (4, 2, 64, 32, True, 127, False), (4, 2, 64, 32, True, 128, True),                     # whatever the width: 64 pairs an expert and a tile of tokens
    (8, 2, 64, 36, False, 4096, False)])                                                  # rows of the second product that are no 16-byte multiples
def test_route(experts, top, width, ff, gated, tokens, grouped):
    from cisr_b200.ops import kernels
    h, w = torch.empty(tokens, width, dtype=torch.bfloat16, device="meta"), torch.empty(experts, ff * (2 if gated else 1), width, dtype=torch.bfloat16, device="meta")
    assert kernels.moe_grouped_ok(h, w, top, gated=gated) is grouped
    assert not kernels.moe_grouped_ok(h.float(), w.float(), top, gated=gated)
