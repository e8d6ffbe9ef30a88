"""Single tokens whose keys are one range: the attention kernel writes finished rows, the very numbers of partial sum and merge."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,hq,hkv", [(64, 9, 3), (128, 8, 8), (64, 40, 2)])
@pytest.mark.parametrize("options", [{}, dict(window=33), dict(window=20, keep_first=5), dict(sink=0.5), dict(sink="heads")])
def test_same_bits_as_with_ranges_beyond_the_context(dim, hq, hkv, options):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(dim + hq)
    lens, page = [1, 2, 63, 64, 65, 200, 256, 0], 16
    options = dict(options)
    if options.get("sink") == "heads":
        options["sink"] = torch.linspace(-3, 3, hq, device="cuda")
    window = options.pop("window", None)
    n, width = len(lens), 32
    q = torch.randn(n, hq, dim, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(n * width, hkv, page, dim, generator=g, device="cuda").bfloat16() for _ in range(2))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    table = torch.arange(n * width, dtype=torch.int32, device="cuda").view(n, width)
    outs = []
    for splits in (1, 2):                                  # the second range is empty for every request
        out = torch.full_like(q, float("nan"))
        partial, stats = torch.empty(n, hq, splits, dim, device="cuda"), torch.empty(n, hq, splits, 2, device="cuda")
        assert kernels.attn_decode_finishes(k, v, page, 256, splits) == (splits == 1)
        kernels.attn_decode(q, out, k, v, i32(range(n)), table, i32(range(n)), n, i32(range(n)), i32(lens), partial, stats, hq, hkv, page, dim ** -0.5, window, 256,
                            splits, staging="tensor_map", **options)
        outs.append(out)
    kernels.raise_if_kernel_gave_up()
    assert not outs[0].isnan().any() and torch.equal(*outs) and (outs[0][-1] == 0).all() and outs[0][:-1].abs().sum((1, 2)).gt(0).all()
