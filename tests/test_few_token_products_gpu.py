"""The tcgen05 products of few tokens with large matrices (csrc/few_gemm.cu), and which calls go there."""
import math

import pytest
import torch

from cisr_b200.ops import kernels
from cisr_b200.parts import linear as products

# rows and K: fewer rows than a block, half a block of K, one share and 2, 4 and 8 of them, uneven ones
SIZES = [(49, 64), (100, 192), (4000, 576), (576, 1536), (300, 2112), (20000, 1024), (1030, 8256)]


def close(got, want, k, scale):
    """Float sums of k products of bfloat16 values with |w| ~ scale, |a| ~ 1: k roundings of 2^-24 of the partial sums, which stay below 6 sigma."""
    bound = k * 2.0 ** -24 * 6 * math.sqrt(k) * scale + 1e-6
    assert float((got.double() - want).abs().max()) <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", SIZES)
@pytest.mark.parametrize("tokens", [1, 5, 16])
def test_plain(n, k, tokens):
    g = torch.Generator().manual_seed(n + k + tokens)
    w = (0.1 * torch.randn(n, k, generator=g)).bfloat16()
    a = torch.randn(tokens, k, generator=g).bfloat16()
    want = a.double() @ w.double().T
    out = torch.full((tokens + 1, n), 7.0, device="cuda")
    kernels.skinny_gemm(w.cuda(), tokens, act=a.cuda(), out=out, kind="few")
    close(out[:tokens].cpu(), want, k, 0.1)
    assert bool((out[tokens:] == 7).all())                              # rows beyond the tokens stay
    before = torch.randn(tokens, n, generator=g)
    added = before.cuda()
    kernels.skinny_gemm(w.cuda(), tokens, act=a.cuda(), out=added, kind="few", accumulate=True)
    assert torch.equal(added.cpu(), before + out[:tokens].cpu())
    kernels.raise_if_kernel_gave_up()


@pytest.mark.gpu
@pytest.mark.parametrize("gate,limit", [("silu", None), ("gelu_tanh", None), ("gated_clamp", 1.5)])
@pytest.mark.parametrize("inter,k", [(7, 64), (200, 320), (1000, 2112), (10000, 576)])
def test_gated(gate, limit, inter, k):
    g = torch.Generator().manual_seed(inter + k)
    w = (torch.randn(2 * inter, k, generator=g) * k ** -0.5).bfloat16().cuda()
    for tokens in (1, 9, 16):
        a = torch.randn(tokens, k, generator=g).bfloat16().cuda()
        sums = torch.empty(tokens, 2 * inter, device="cuda")
        kernels.skinny_gemm(w, tokens, act=a, out=sums, kind="few")
        want = torch.empty(tokens, inter, dtype=torch.bfloat16, device="cuda")
        kernels.swiglu(sums, want, gate=gate, limit=limit)
        got = torch.full((tokens, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
        kernels.skinny_gemm(w, tokens, act=a, epilogue=kernels.EPI_SWIGLU, out=got, kind="few", gate=gate, gate_limit=limit)
        # the same float sums up to their order, then one rounding to bfloat16: at most a step apart
        torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -7, atol=1e-5)
    kernels.raise_if_kernel_gave_up()


@pytest.mark.gpu
@pytest.mark.parametrize("dim,hq,hkv", [(64, 9, 3), (64, 2, 1), (128, 2, 1), (128, 32, 8)])
@pytest.mark.parametrize("tokens", [1, 11, 16])
def test_rotation_and_cache(dim, hq, hkv, tokens):
    page, hidden = 4, 576
    g = torch.Generator().manual_seed(dim * hq + tokens)
    w = (0.1 * torch.randn((hq + 2 * hkv) * dim, hidden, generator=g)).bfloat16().cuda()
    a = torch.randn(tokens, hidden, generator=g).bfloat16().cuda()
    positions = torch.randperm(40, generator=g)[:tokens].to(torch.int32).cuda()
    token_req = (torch.arange(tokens) % 3).to(torch.int32).cuda()
    req_slot = torch.tensor([2, 0, 1], dtype=torch.int32, device="cuda")
    table = torch.arange(36, dtype=torch.int32).reshape(3, 12).cuda()
    table[1, 5:] = -1                                                   # a slot without those pages: its tokens write no keys
    angles = torch.randn(tokens, dim // 2, generator=g).cuda()
    cos, sin = angles.cos(), angles.sin()
    sums = torch.empty(tokens, w.shape[0], device="cuda")
    kernels.skinny_gemm(w, tokens, act=a, out=sums, kind="few")
    results = []
    for fused in (False, True):
        q = torch.zeros(tokens, hq, dim, dtype=torch.bfloat16, device="cuda")
        kc = torch.zeros(36, hkv, page, dim, dtype=torch.bfloat16, device="cuda"); vc = torch.zeros_like(kc)
        if fused:
            kernels.skinny_gemm(w, tokens, act=a, epilogue=kernels.EPI_ROPE, kind="few",
                                rope=dict(cos=cos, sin=sin, rot_half=dim // 2, interleaved=False, q_out=q, k_cache=kc, v_cache=vc, positions=positions,
                                          token_req=token_req, req_slot=req_slot, block_table=table, page_size=page, hq=hq, hkv=hkv, dim=dim))
        else:
            kernels.rope_store(sums, hq * dim, (hq + hkv) * dim, cos, sin, dim // 2, False, q, kc, vc, token_req, positions, req_slot, table, page,
                               hq, hkv, dim)
        results.append((q.float(), kc.float(), vc.float()))
    for got, want in zip(results[1], results[0]):
        assert float(got.abs().sum()) > 0
        # sums of the same shares up to their order (2^-24 of them each) and one rounding to bfloat16
        torch.testing.assert_close(got, want, rtol=2.0 ** -7, atol=1e-5)
        assert torch.equal(got == 0, want == 0)
    kernels.raise_if_kernel_gave_up()


@pytest.mark.gpu
def test_calls_that_go_elsewhere():
    w = torch.randn(200, 96, device="cuda").bfloat16()
    a, out = torch.randn(4, 96, device="cuda").bfloat16(), torch.empty(4, 200, device="cuda")
    with pytest.raises(kernels.KernelError, match="few_gemm"):
        kernels.skinny_gemm(w, 4, act=a, out=out, kind="few")           # K in no whole groups of 64
    w = torch.randn(200, 128, device="cuda").bfloat16()
    with pytest.raises(kernels.KernelError, match="few_gemm"):
        kernels.skinny_gemm(w, 4, x=torch.randn(4, 128, device="cuda"), norm_w=torch.ones(128, device="cuda"), out=out, kind="few")


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [1, 12])
def test_long_rows_and_misaligned_activations(tokens):
    g = torch.Generator().manual_seed(tokens)
    w = (0.1 * torch.randn(300, 14336, generator=g)).bfloat16()
    flat = torch.randn(tokens * 14336 + 1, generator=g).bfloat16().cuda()
    for a in (flat[:-1].view(tokens, 14336), flat[1:].view(tokens, 14336)):
        close(products.linear(a, w.cuda()).cpu(), a.cpu().double() @ w.double().T, 14336, 0.1)


def test_rule():
    w = torch.empty(8192, 576, dtype=torch.bfloat16, device="meta")
    big = torch.empty(4096, 14336, dtype=torch.bfloat16)
    assert kernels.few_takes(1, big) and kernels.few_takes(16, big) and not kernels.few_takes(17, big) and not kernels.few_takes(0, big)
    assert not kernels.few_takes(4, w[:1024]) and not kernels.few_takes(4, big.float()[:, :64])
    assert not kernels.few_takes(4, big.view(-1)[:8192 * 1000].view(8192, 1000))                     # K in no whole groups of 64
    assert not kernels.few_takes(4, big.view(-1)[4:4 + 4096 * 4096].view(4096, 4096))                # rows that start off 16 bytes
    assert kernels.few_takes(4, big, (128, 64, False)) and kernels.few_takes(4, big, (64, 32, False))
    for turn in ((128, 64, True), (128, 32, False), (96, 48, False), (128, 0, False)):
        assert not kernels.few_takes(4, big, turn)
    assert kernels.skinny_ok(16, big) and not kernels.skinny_ok(16, big, (96, 48, False))


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(49152, 576), (8192, 2048), (4096, 4096), (1024, 4160)])
@pytest.mark.parametrize("tokens", [1, 16])
def test_sums_are_as_exact_as_the_streaming_kernels(n, k, tokens):
    """The tensor core cuts what it adds: with K in one accumulator these sums were 3.6 times (K 576) and 4.5 times (K 2048) as far from 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(k)
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    a = torch.randn(tokens, k, generator=g, device="cuda").bfloat16()
    want, errors = a.double() @ w.double().T, {}
    for kind in ("few", "stream"):
        out = torch.empty(tokens, n, device="cuda")
        kernels.skinny_gemm(w, tokens, act=a, out=out, kind=kind)
        errors[kind] = float((out.double() - want).norm() / want.norm())
    kernels.raise_if_kernel_gave_up()
    assert errors["few"] <= 1.1 * errors["stream"], errors           # the same number of cuts; a tenth for how they fall
