"""The tcgen05 products of one round of CTAs: tile widths, row tiles and shares of K at the edges of their rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(m, n, kk):
    g = torch.Generator(device="cuda").manual_seed(m + n + kk)
    a, w = (torch.randn(r, kk, generator=g, device="cuda").bfloat16() for r in (m, n))
    return a, w, a.double() @ w.double().T


def near(got, want, kk):
    # kk float additions of products of size 1, in shares of K, and the rounding of the result
    assert ((got.double() - want).abs() <= 8e-6 * kk ** 0.5 + 1e-5 * want.abs()).all()


@pytest.mark.parametrize("m,n,kk", [(1, 66, 1472), (200, 576, 1536), (300, 4736, 1536), (257, 64, 2048), (129, 33, 2056),  # 64 columns, K in 1 and 2
                                    (64, 4096, 4096), (128, 4737, 2056), (130, 9472, 2120), (700, 300, 4104),               # 128: 4, 2 and 1
                                    (129, 9600, 520), (900, 4500, 200), (256, 18944, 72), (100, 19000, 520), (256, 18945, 520), (90, 37900, 72)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_plain(m, n, kk, accumulate):
    from cisr_b200.ops import kernels
    a, w, want = operands(m, n, kk)
    out = torch.ones(m, n, device="cuda") if accumulate else torch.full((m, n), float("nan"), device="cuda")
    kernels.gemm_tcgen05(a, w, out, accumulate, 0.5)
    kernels.raise_if_kernel_gave_up()
    near(out, 0.5 * want + accumulate, kk)


@pytest.mark.parametrize("m,inter,kk", [(200, 1500, 576), (64, 2368, 1536), (128, 2000, 4096), (200, 4800, 520), (900, 2300, 200), (100, 9500, 520), (256, 9500, 136),
                                       (1000, 4800, 520), (1000, 4800, 768), (1000, 4800, 776), (2100, 700, 576)])       # more than one round: K to 768 and beyond
@pytest.mark.parametrize("gate", ["silu", "gelu_tanh", "gated_clamp"])
def test_gated(m, inter, kk, gate):
    from cisr_b200.ops import kernels
    a, w, _ = operands(m, 2 * inter, kk)
    w = (w.float() * (4 * kk ** -0.5)).bfloat16()
    z = a.double() @ w.double().T
    x, u = z[:, :inter], z[:, inter:]
    if gate == "gated_clamp":
        x, u = x.clamp(max=7.0), u.clamp(-7.0, 7.0)
        want = x * torch.sigmoid(1.702 * x) * (u + 1)
    else:
        want = (torch.nn.functional.silu(x) if gate == "silu" else torch.nn.functional.gelu(x, approximate="tanh")) * u
    out = torch.full((m, inter), float("nan"), device="cuda", dtype=torch.bfloat16)
    kernels.gemm_tcgen05_swiglu(a, w, out, gate, 7.0 if gate == "gated_clamp" else None)
    kernels.raise_if_kernel_gave_up()
    assert ((out.double() - want).abs() <= 1e-3 + 2 ** -7 * want.abs()).all()       # bfloat16's 2^-9 with room for the sums' error


@pytest.mark.parametrize("m,hq,hkv,dim,kk", [(200, 9, 3, 64, 576), (64, 32, 8, 128, 4096), (130, 8, 8, 64, 4104), (200, 16, 4, 128, 2048), (200, 66, 5, 128, 520), (700, 32, 8, 128, 200)])
def test_rotated(m, hq, hkv, dim, kk):
    from cisr_b200.ops import kernels
    a, w, _ = operands(m, (hq + 2 * hkv) * dim, kk)
    w = (w.float() * kk ** -0.5).bfloat16()
    z = (a.double() @ w.double().T).view(m, -1, dim)
    angle = torch.arange(m, device="cuda", dtype=torch.float64)[:, None] * 100.0 ** (-torch.arange(dim // 2, device="cuda", dtype=torch.float64) / dim)
    cos, sin = angle.cos(), angle.sin()
    x, y = z[:, :hq + hkv, :dim // 2], z[:, :hq + hkv, dim // 2:]
    c, s = cos[:, None], sin[:, None]
    turned = torch.cat([torch.cat([x * c - y * s, y * c + x * s], -1), z[:, hq + hkv:]], 1)
    order = torch.randperm(m, device="cuda").int()
    q = torch.full((m, hq, dim), float("nan"), device="cuda", dtype=torch.bfloat16)
    caches = [torch.full((-(-m // 16), hkv, 16, dim), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    zero = torch.zeros(m, dtype=torch.int32, device="cuda")
    kernels.gemm_tcgen05_rope(a, w, dict(cos=cos.float(), sin=sin.float(), q_out=q, k_cache=caches[0], v_cache=caches[1], positions=order, token_req=zero,
                                         req_slot=zero[:1], block_table=torch.arange(-(-m // 16), dtype=torch.int32, device="cuda")[None], page_size=16,
                                         hq=hq, hkv=hkv, dim=dim))
    kernels.raise_if_kernel_gave_up()
    for got, want in ((q, turned[:, :hq]), *((cache.transpose(1, 2).reshape(-1, hkv, dim)[order.long()], turned[:, at:at + hkv])
                                             for cache, at in zip(caches, (hq, hq + hkv)))):
        assert ((got.double() - want).abs() <= 1e-3 + 2 ** -8 * want.abs()).all()


@pytest.mark.parametrize("m,inter,kk", [(130, 200, 64), (1000, 4800, 64), (1000, 4800, 2056)])
@pytest.mark.parametrize("gate,x,up", [("silu", -88.0, 1e30), ("silu", -87.5, 1e30), ("gelu_tanh", -10.0, 1e30), ("gated_clamp", -51.75, 3.0)])
def test_quotients_of_large_denominators(gate, x, up, m, inter, kk):
    """1 + exp(.) above 2^126: the gate is small and not zero."""
    from cisr_b200.ops import kernels
    a, w = torch.zeros(m, kk, device="cuda", dtype=torch.bfloat16), torch.zeros(2 * inter, kk, device="cuda", dtype=torch.bfloat16)
    a[:, 0] = 1
    w[:inter, 0], w[inter:, 0] = x, up
    z, u = (torch.tensor(v).bfloat16().double() for v in (x, up))
    if gate == "gelu_tanh":
        want = z / (1 + torch.exp(-2 * 0.7978845608028654 * (z + 0.044715 * z ** 3))) * u
    else:
        want = z * torch.sigmoid(1.702 * z) * (u + 1) if gate == "gated_clamp" else z * torch.sigmoid(z) * u
    out = torch.full((m, inter), float("nan"), device="cuda", dtype=torch.bfloat16)
    kernels.gemm_tcgen05_swiglu(a, w, out, gate, 7.0 if gate == "gated_clamp" else None)
    kernels.raise_if_kernel_gave_up()
    # the exponential carries a few 2^-24 of its argument of 88 (1e-4 with room), the result bfloat16's rounding of eight bits, 2^-8
    assert ((out.double() - want).abs() <= (2 ** -8 + 1e-4) * want.abs()).all()
