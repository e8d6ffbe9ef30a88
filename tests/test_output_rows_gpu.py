"""Norm, weight and gate of the recurrences' read-outs four columns at a time, at the edges of their runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOLERANCE = {torch.float32: 3e-6, torch.bfloat16: 2 ** -8}      # some twenty roundings of 2^-24; one of 2^-9 on top


def gated(normed, gate, w):
    return normed * w.double() * torch.sigmoid(gate.double())


def drawn(seed, *shapes):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*s, generator=g, device="cuda") for s in shapes]


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,width,pad", [(3, 508, 0), (3, 512, 4), (130, 1028, 4), (2, 2048, 0), (5, 4096, 8), (2, 4100, 0), (2, 1026, 2)])
def test_whole_rows(out_dtype, tokens, width, pad):
    from cisr_b200.ops import kernels
    o, gate, w = drawn(width, (tokens, width), (tokens, width + 8), (width,))
    out = torch.full((tokens, width + pad), 5.0, dtype=out_dtype, device="cuda")
    kernels.lightning_output(o, gate, 4, w, 1e-5, out)
    want = gated(o.double() * torch.rsqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5), gate[:, 4:4 + width], w)
    assert ((out[:, :width].double() - want).abs() <= TOLERANCE[out_dtype] * want.abs() + 1e-30).all() and (out[:, width:] == 5.0).all()


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,dv", [(3, 2, 124), (5, 3, 128), (33, 4, 256), (2, 2, 260), (7, 1, 512), (2, 2, 516), (2, 2, 130)])
def test_heads(out_dtype, tokens, heads, dv):
    from cisr_b200.ops import kernels
    y, yn, m, gate, w = drawn(dv, (tokens, heads * dv), (tokens, heads), (tokens, heads), (tokens, heads * dv + 8), (heads * dv,))
    out = torch.full((tokens, heads * dv), 5.0, dtype=out_dtype, device="cuda")
    kernels.exp_output(y.view(tokens, heads, dv), yn, m, gate, 4, w, 1e-3, out)
    o = y.double().view(tokens, heads, dv) / (torch.maximum(yn.double().abs(), torch.exp(-m.double())) + 1e-6)[..., None]
    want = gated((o * torch.rsqrt((o ** 2).mean(-1, keepdim=True) + 1e-3)).view(tokens, -1), gate[:, 4:4 + heads * dv], w)
    assert ((out.double() - want).abs() <= TOLERANCE[out_dtype] * want.abs() + 1e-30).all()


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gates_of_large_denominators(out_dtype):
    """1 + exp(-gate) above 2^126: the gate is small and not zero."""
    from cisr_b200.ops import kernels
    tokens, heads, dv = 3, 4, 128
    width = heads * dv
    (o,) = drawn(1, (tokens, width))
    gate, w = torch.full((tokens, width), -88.0, device="cuda"), torch.full((width,), 1e30, device="cuda")
    out = torch.empty(tokens, width, dtype=out_dtype, device="cuda")
    kernels.lightning_output(o, gate, 0, w, 1e-5, out)
    want = gated(o.double() * torch.rsqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5), gate, w)
    tolerance = TOLERANCE[out_dtype] + 1e-5                              # and 2^-24 of the exponent 88
    assert ((out.double() - want).abs() <= tolerance * want.abs()).all()
    yn, m = torch.full((tokens, heads), 2.0, device="cuda"), torch.zeros(tokens, heads, device="cuda")
    kernels.exp_output(o.view(tokens, heads, dv), yn, m, gate, 0, w, 1e-5, out)
    v = o.double().view(tokens, heads, dv) / (2 + 1e-6)
    want = gated((v * torch.rsqrt((v ** 2).mean(-1, keepdim=True) + 1e-5)).view(tokens, width), gate, w)
    assert ((out.double() - want).abs() <= tolerance * want.abs()).all()
