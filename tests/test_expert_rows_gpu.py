"""Routed experts for many tokens: the sort and the combining kernel at the edges of their batches, against plain indexing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top,experts", [(1, 1, 1), (130, 4, 33), (4096, 4, 64), (5000, 7, 100), (300, 2, 3)])
def test_sort_places_every_pair_once(tokens, top, experts):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(tokens)
    chosen = torch.randint(0, experts + 2, (tokens, top), generator=g, device="cuda", dtype=torch.int32)      # two outputs have no matrices
    rows = kernels.moe_sorted_rows(tokens, top, experts)
    row_of, src, group = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (tokens * top, rows, rows // kernels.MOE_TILE))
    kernels.moe_sort(chosen, experts, row_of, src, group)
    flat, row = chosen.reshape(-1).long(), row_of.long()
    real = flat < experts
    assert (row[~real] == -1).all() and row[real].unique().numel() == int(real.sum())
    assert torch.equal(src.long()[row[real]], torch.arange(tokens * top, device="cuda")[real] // top) and int((src >= 0).sum()) == int(real.sum())
    assert torch.equal(group.long()[row[real] // kernels.MOE_TILE], flat[real])
    counts = torch.bincount(flat[real], minlength=experts)
    assert int((group >= 0).sum()) == int(((counts + kernels.MOE_TILE - 1) // kernels.MOE_TILE).sum())


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("tokens,top,hidden", [(3, 1, 4), (5, 7, 1028), (17, 8, 4096), (4, 64, 36), (4, 65, 36), (6, 3, 30)])
def test_combine(tokens, top, hidden, scaled):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(top + hidden)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    rows, weight, h, scale = rand(50, hidden), rand(tokens, top), rand(tokens, hidden).bfloat16(), rand(hidden)
    row_of = torch.randint(-1, 50, (tokens * top,), generator=g, device="cuda", dtype=torch.int32)
    picked = torch.where(row_of[:, None] >= 0, rows[row_of.clamp(min=0).long()].double(), h.double().repeat_interleave(top, 0)).view(tokens, top, hidden)
    want = (weight.double()[..., None] * picked).sum(1) * (scale.double() if scaled else 1.0)
    out = torch.full((tokens, hidden), float("nan"), device="cuda")
    kernels.moe_combine(rows, row_of, weight, out, scale if scaled else None, h=h)
    assert float((out.double() - want).norm() / want.norm()) < 1e-6      # `top` float multiply-adds, 2^-24 each
