"""Float prompt attention by products of split floats: edges of its 32-query and 64- or 32-key tiles, every kind of mask, numbers that are not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def attend(portions, dim, hq, hkv, page=16, window=None, keep_first=0, sink=None, softcap=None, change=None):
    """(the kernel's output, the same in 64 bits) for portions of (tokens, keys before them)."""
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(dim + hq + sum(n + 7 * b for n, b in portions))
    tokens, ctx = sum(n for n, _ in portions), [n + b for n, b in portions]
    q = torch.randn(tokens, hq, dim, generator=g, device="cuda")
    width = -(-max(ctx) // page)
    pages = width * len(portions) + 1
    k, v = (torch.randn(pages, hkv, page, dim, generator=g, device="cuda") for _ in range(2))
    table = (torch.randperm(pages - 1, generator=torch.Generator().manual_seed(3))[: width * len(portions)] + 1).int().cuda().view(len(portions), width)
    if change:
        change(q, k, v, table)
    out = torch.full_like(q, float("nan"))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    tiles = [(r, q0) for r, (n, _) in enumerate(portions) for q0 in range((n - 1) // 64 * 64, -1, -64)]
    starts = [sum(n for n, _ in portions[:r]) for r in range(len(portions))]
    kernels.attn_prefill(q, out, k, v, i32(range(len(portions))), table, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), i32(starts),
                         i32([n for n, _ in portions]), i32(ctx), hq, hkv, page, dim ** -0.5, window, sink=sink, keep_first=keep_first, softcap=softcap)
    want = []
    for r, (n, before) in enumerate(portions):
        keys, values = (x[table[r].long()].transpose(1, 2).reshape(-1, hkv, dim)[:ctx[r]].double().nan_to_num(0.0, float("inf"), float("-inf")).repeat_interleave(hq // hkv, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[starts[r]:starts[r] + n].double(), keys) * dim ** -0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        at, key = torch.arange(before, before + n, device="cuda")[:, None], torch.arange(ctx[r], device="cuda")
        seen = key <= at
        if window:
            seen &= (at - key < window) | (key < keep_first)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat((s, torch.as_tensor(sink, dtype=torch.float64, device="cuda").expand(hq)[:, None, None].expand(hq, n, 1)), -1)
        p = torch.softmax(s, -1)[..., :ctx[r]]
        want.append(torch.einsum("hqk,khd->qhd", p, torch.where(p.sum((0, 1))[:, None, None] > 0, values, 0.0)))
    return out, torch.cat(want)


def near(got, want):
    # scores of a few units carry 2^-23 of themselves into the exponential, and as much comes of the sums
    assert ((got.double() - want).abs() <= 3e-6 * (1 + want.abs())).all()


@pytest.mark.parametrize("portions", [[(2, 0)], [(31, 0), (32, 0), (33, 0)], [(64, 63), (65, 64)], [(97, 1000)], [(300, 0), (2, 130)]])
@pytest.mark.parametrize("dim,hq,hkv", [(16, 3, 1), (48, 2, 2), (64, 6, 2), (128, 4, 1)])
def test_edges(portions, dim, hq, hkv):
    near(*attend(portions, dim, hq, hkv))


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("options", [dict(window=1), dict(window=40), dict(window=64, keep_first=3), dict(window=100, keep_first=70), dict(sink=0.5), dict(page=8, window=33)])
def test_masks(dim, options):
    near(*attend([(200, 0), (70, 333)], dim, 4, 2, **options))


def test_sink_per_head_and_bent_scores():
    near(*attend([(90, 20)], 64, 4, 2, sink=torch.tensor([0.0, -3.0, 5.0, float("-inf")], device="cuda")))
    near(*attend([(90, 20)], 64, 4, 2, softcap=2.0))


@pytest.mark.parametrize("what", [float("inf"), float("-inf"), 3.4e38])
def test_scores_without_bound(what):
    """A key whose scores are infinite: -inf is a weight of zero, not NaN; every row that does not see it stays as it was."""
    def change(q, k, v, table):
        q[..., 0] = -q[..., 0].abs() - 1 if what > 0 else q[..., 0].abs() + 1
        k[table[0, 2].item(), :, 5, 0] = what         # key 37 has the score -inf (or so low that its weight is 0) for every query
        k[table[0, 2].item(), :, 5, 1:] = 0
    near(*attend([(120, 0)], 64, 4, 2, change=change))


def test_values_without_bound():
    def change(q, k, v, table):
        v[table[0, 4].item(), :, 7, 3] = float("nan")          # key 71
    got, want = attend([(120, 0)], 64, 4, 2, change=change)
    bad = torch.zeros_like(got, dtype=torch.bool)
    bad[71:, :, 3] = True
    assert got[bad].isnan().all()
    near(got[~bad], want[~bad])


@pytest.mark.parametrize("power", [-60, -100, -112, -120])
def test_small_values(power):
    """Values whose bfloat16 parts run out of exponents."""
    got, want = attend([(70, 33), (5, 0)], 64, 4, 2, change=lambda q, k, v, table: v.abs_().mul_(2.0 ** power))
    # as `near`, and the rounding of a probability's product with a value to the last place of a subnormal, 103 keys
    assert ((got.double() - want).abs() <= 6e-6 * want + 103 * 2.0 ** -149).all()
