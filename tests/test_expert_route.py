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


@pytest.mark.parametrize("tokens,top,experts,width,ff", [(16, 8, 64, 64, 32), (1, 2, 4, 64, 32), (300, 4, 8, 64, 48)])
def test_scratch_is_a_row_per_pair(tokens, top, experts, width, ff, monkeypatch):
    """Padded to whole tiles, 16 tokens of 64 experts held 206 MB for 3 MB of rows at a width of 4096."""
    from cisr_b200.ops import kernels
    rows, tiles = [], []
    monkeypatch.setattr(kernels, "_need", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "moe_sort", lambda chosen, experts, row_of, src, group, t, n: (rows.append(n), tiles.append(t)))
    monkeypatch.setattr(kernels, "moe_scatter", lambda h, row_of, out: rows.append(out.shape[0]) or out)
    monkeypatch.setattr(kernels, "gemm_tcgen05_experts", lambda a, w, out, *rest: rows.append(out.shape[0]) or out)
    monkeypatch.setattr(kernels, "moe_combine", lambda rows_out, row_of, weight, out, scale, h: out)
    t = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    kernels.moe_grouped(t(tokens, width), t(experts, 2 * ff, width), t(experts, width, ff), torch.zeros(tokens, top, dtype=torch.int32),
                        torch.zeros(tokens, top), torch.zeros(tokens, width), gate_limit=7.0)
    assert rows == [tokens * top] * 4 and tiles[0].shape == (kernels.moe_tiles(tokens, top, experts), 4)


def test_what_the_products_by_expert_do_not_take_stays_with_the_rows():
    """Buffers that start off a 16-byte boundary, and more experts than the sort has room for, took `moe_rows` before few tokens were sorted."""
    from cisr_b200.ops import kernels
    off = lambda *s: torch.zeros(torch.Size(s).numel() + 1, dtype=torch.bfloat16)[1:].view(*s)
    meta = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device="meta")
    h, up, down = meta(64, 1024), meta(16, 768, 1024), meta(16, 1024, 384)
    assert kernels.moe_grouped_ok(h, up, 4, gated=True, w_down=down)
    assert not kernels.moe_grouped_ok(off(64, 1024), up, 4, gated=True, w_down=down)
    assert not kernels.moe_grouped_ok(h, off(16, 768, 1024), 4, gated=True, w_down=down)
    assert not kernels.moe_grouped_ok(h, up, 4, gated=True, w_down=off(16, 1024, 384))
    most = kernels.MOE_SORT_MAX_EXPERTS
    assert kernels.moe_grouped_ok(meta(4096, 64), meta(most, 64, 64), 128) and not kernels.moe_grouped_ok(meta(4096, 64), meta(most + 1, 64, 64), 128)
