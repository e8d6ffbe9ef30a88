"""The gated feed-forward of few tokens launched by one call: the same as its two products, and the calls it does not take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 4, 8, 9, 16])
@pytest.mark.parametrize("k,inter,n", [(576, 1536, 576), (72, 40, 24), (1024, 1000, 640)])
@pytest.mark.parametrize("gate", ["silu", "gelu_tanh", "gated_clamp"])
def test_same_as_two_products(tokens, k, inter, n, gate):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(tokens + k)
    h, gate_up, down = ((torch.randn(*s, generator=g, device="cuda") * s[1] ** -0.5).bfloat16() for s in ((tokens, k), (2 * inter, k), (n, inter)))
    limit = 0.7 if gate == "gated_clamp" else None
    act, want = torch.empty(tokens, inter, device="cuda", dtype=torch.bfloat16), torch.empty(tokens, n, device="cuda")
    kernels.skinny_gemm(gate_up, tokens, act=h, epilogue=kernels.EPI_SWIGLU, out=act, gate=gate, gate_limit=limit)
    kernels.skinny_gemm(down, tokens, act=act, epilogue=kernels.EPI_PLAIN, out=want)
    assert kernels.skinny_mlp_ok(h, gate_up, down)
    assert torch.equal(kernels.skinny_mlp(h, gate_up, down, gate, limit), want)


def test_what_it_leaves_to_others():
    from cisr_b200.ops import kernels
    h, gate_up, down = (torch.zeros(*s, device="cuda", dtype=torch.bfloat16) for s in ((4, 576), (3072, 576), (576, 1536)))
    assert not kernels.skinny_mlp_ok(h.new_zeros(17, 576), gate_up, down) and not kernels.skinny_mlp_ok(h.float(), gate_up, down)
    assert not kernels.skinny_mlp_ok(h, h.new_zeros(8192, 576), h.new_zeros(576, 4096)) and not kernels.skinny_mlp_ok(h[:0], gate_up, down)
    with pytest.raises(kernels.KernelError):
        kernels.skinny_mlp(h, gate_up, down[:, :1528].contiguous())
    with pytest.raises(kernels.KernelError):
        kernels.skinny_mlp(h, gate_up, down, "gated_clamp")


def test_activations_off_a_16_byte_boundary():
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(3)
    flat, gate_up, down = ((torch.randn(*s, generator=g, device="cuda") * 576 ** -0.5).bfloat16() for s in ((4 * 576 + 8,), (3072, 576), (576, 1536)))
    for start in (1, 4, 7):
        h = flat[start:start + 4 * 576].view(4, 576)
        assert h.data_ptr() % 16 and torch.equal(kernels.skinny_mlp(h, gate_up, down), kernels.skinny_mlp(h.clone(), gate_up, down))
