"""Products of rows sorted by expert, weight rows on the lanes: edges of the runs, ragged widths, every epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu
COUNTS = [[0, 1, 15, 16, 17], [31, 32, 33, 0, 63], [255, 256, 257, 0, 0, 5], [700, 1, 513], [0, 0, 129], [1] * 40]


def sorted_rows(counts, k, seed):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(seed)
    experts, pairs = len(counts), sum(counts)
    chosen = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))
    chosen = chosen[torch.randperm(pairs, generator=torch.Generator().manual_seed(seed))].int().cuda().view(pairs, 1)
    rows = kernels.moe_sorted_rows(pairs, 1, experts)
    row_of = torch.empty(pairs, dtype=torch.int32, device="cuda")
    tiles = torch.full((kernels.moe_tiles(pairs, 1, experts), 4), -7, dtype=torch.int32, device="cuda")
    kernels.moe_sort(chosen, experts, row_of, None, None, tiles, rows)
    h = torch.randn(pairs, k, generator=g, device="cuda").bfloat16()
    a = kernels.moe_scatter(h, row_of, torch.full((rows, k), float("nan"), device="cuda", dtype=torch.bfloat16))      # what lies between the runs is not read
    return g, chosen.flatten().long(), row_of.long(), tiles, h, a


@pytest.mark.parametrize("counts", COUNTS)
def test_runs(counts):
    from cisr_b200.ops import kernels
    _, chosen, row_of, tiles, _, _ = sorted_rows(counts, 8, 1)
    seen, got = [], tiles.tolist()
    used = [t for t in got if t[2]]
    assert got[:len(used)] == used and all(t == [0, 0, 0, 0] for t in got[len(used):]) and all(t[2] <= kernels.MOE_RUN for t in used)
    for expert, first, rows, _ in used:
        seen += [(first + i, expert) for i in range(rows)]
    assert sorted(seen) == sorted(zip(row_of.tolist(), chosen.tolist()))


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("n,k", [(512, 264), (300, 72), (128, 1096)])
@pytest.mark.parametrize("kind", ["plain", "relu_squared", "gelu", "gated"])
def test_products(counts, n, k, kind):
    from cisr_b200.ops import kernels
    g, chosen, row_of, tiles, h, a = sorted_rows(counts, k, n + k)
    n -= n % 8 if kind == "gated" else 0
    w = (torch.randn(len(counts), n * (2 if kind == "gated" else 1), k, generator=g, device="cuda") * (3 * k ** -0.5)).bfloat16()
    out = torch.full((a.shape[0], n), float("nan"), device="cuda", dtype=torch.float32 if kind == "plain" else torch.bfloat16)
    kernels.gemm_tcgen05_experts(a, w, out, tiles, None, "relu_squared" if kind in ("plain", "gated") else kind, 4.0 if kind == "gated" else None)
    kernels.raise_if_kernel_gave_up()
    z = torch.einsum("pk,pnk->pn", h.double(), w.double()[chosen])
    if kind == "relu_squared":
        z = z.clamp(min=0) ** 2
    elif kind == "gelu":
        z = torch.nn.functional.gelu(z)
    elif kind == "gated":
        gate, up = z[:, :n].clamp(max=4.0), z[:, n:].clamp(-4.0, 4.0)
        z = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    got = out[row_of].double()
    # k float additions of products of size 3 k^-1/2, and the rounding of a bfloat16 result
    assert ((got - z).abs() <= (3e-5 if kind == "plain" else 1e-3 + 2 ** -8 * z.abs()) + 1e-5 * z.abs()).all()
    rest = torch.ones(a.shape[0], dtype=torch.bool, device="cuda")
    rest[row_of] = False
    assert out[rest].isnan().all()                       # rows outside the runs are not written


@pytest.mark.parametrize("experts", [3072, 3073, 4096, 12288])      # counts of up to 48 KB, and beyond
def test_sort_of_many_experts(experts):
    from cisr_b200.ops import kernels
    chosen = torch.randint(0, experts, (500, 3), generator=torch.Generator().manual_seed(experts)).int()
    row_of, tiles = torch.empty(1500, dtype=torch.int32, device="cuda"), torch.empty(kernels.moe_tiles(500, 3, experts), 4, dtype=torch.int32, device="cuda")
    kernels.moe_sort(chosen.cuda(), experts, row_of, None, None, tiles, 1500)
    assert torch.equal(chosen.flatten()[torch.argsort(row_of.cpu())].long(), chosen.flatten().long().sort().values) and row_of.unique().numel() == 1500
    assert int(tiles[:, 2].sum()) == 1500
