"""The delta rule's row kernels on both sides of their dispatch rules, against the same steps in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device="cuda")


# the tile kernel takes more than 64 tokens, four taps, whole runs of four channels and q and k channels that fit 48 KB with its
# indices (3072 do not); portions begin at every place of its tiles of four tokens and the last tile has one to four tokens
@pytest.mark.parametrize("heads,kvh,dk,dv,taps,lens", [
    (2, 2, 16, 16, 4, [65]), (4, 2, 32, 24, 4, [1, 2, 3, 60, 5]), (3, 1, 12, 8, 4, [7, 64, 2, 1]), (2, 1, 64, 64, 4, [130]),
    (12, 12, 128, 16, 4, [66]), (16, 16, 96, 8, 4, [70]), (11, 11, 128, 16, 4, [3, 66]), (24, 24, 64, 8, 4, [80]),      # 3072, 3072, 2816, 3072 q and k channels
    (2, 2, 16, 16, 4, [64]), (2, 2, 16, 16, 3, [66]), (2, 1, 7, 5, 4, [66])])
def test_prepare(heads, kvh, dk, dv, taps, lens):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(dk + dv + len(lens))
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T, channels, matrix = sum(lens), 2 * kvh * dk + heads * dv, heads * dk * dv
    cols = -(-(channels + heads * dv + 2 * heads) // 4) * 4
    proj, conv_w, state = rand(T, cols), rand(channels, taps), rand(len(lens), matrix + (taps - 1) * channels)
    a_log, dt_bias = rand(heads), rand(heads)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    slots = list(reversed(range(len(lens))))
    req = [r for r, n in enumerate(lens) for _ in range(n)]
    qkv, beta, decay = (torch.full((T, w), float("nan"), device="cuda") for w in (channels, heads, heads))
    kernels.delta_prepare(proj, conv_w, taps, state, a_log, dt_bias, i32(req), i32(slots), i32(starts), qkv, beta, decay, heads, kvh, dk, dv, 1e-6)
    P = proj.double()
    want = torch.empty(T, channels, dtype=torch.float64, device="cuda")
    for r, n in enumerate(lens):
        kept = state[slots[r], matrix:].double().view(taps - 1, channels)
        rows = torch.cat([kept, P[starts[r]:starts[r] + n, :channels]])
        want[starts[r]:starts[r] + n] = sum(conv_w[:, j].double() * rows[j:j + n] for j in range(taps))
    want = want * torch.sigmoid(want)
    heads_qk = want[:, :2 * kvh * dk].reshape(T, 2 * kvh, dk)
    unit = heads_qk / torch.sqrt((heads_qk ** 2).sum(-1, keepdim=True) + 1e-6)
    unit[:, :kvh] *= dk ** -0.5
    want[:, :2 * kvh * dk] = unit.reshape(T, -1)
    at = channels + heads * dv
    want_beta = torch.sigmoid(P[:, at:at + heads])
    want_decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(P[:, at + heads:at + 2 * heads] + dt_bias.double()))
    # `taps` multiply-adds, silu and a norm: some ten roundings of 2^-24 of terms of the size of the inputs
    assert ((qkv.double() - want).abs() <= 3e-6 * (1 + want.abs())).all()
    assert ((beta.double() - want_beta).abs() <= 1e-6 * want_beta).all()
    # an exponential carries the error of its argument
    assert ((decay.double() - want_decay).abs() <= 1e-6 * (2 - want_decay.log()) * want_decay + 1e-37).all()


# 8, 16 and 32 lanes share a (token, head), also where its values do not fill them; other widths and strides go to the older kernel
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,dv,gate_col,pad", [(1, 1, 4, 0, 0), (5, 3, 20, 4, 8), (33, 2, 32, 0, 0), (7, 5, 36, 8, 4), (9, 2, 64, 4, 0), (3, 3, 100, 0, 4),
                                                           (17, 2, 128, 4, 0), (3, 2, 132, 4, 0), (4, 2, 33, 4, 0), (4, 2, 64, 2, 0), (4, 2, 64, 4, 2)])
def test_output(out_dtype, tokens, heads, dv, gate_col, pad):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(tokens + dv)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    o, proj, w = rand(tokens, heads, dv), rand(tokens, gate_col + heads * dv + 12 - gate_col % 4), rand(dv)
    out = torch.full((tokens, heads * dv + pad), 5.0, dtype=out_dtype, device="cuda")
    kernels.delta_output(o, proj, gate_col, w, 1e-5, out, heads, dv)
    gate = proj[:, gate_col:gate_col + heads * dv].double().view(tokens, heads, dv)
    unit = o.double() * torch.rsqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    want = (unit * w.double() * gate * torch.sigmoid(gate)).view(tokens, -1)
    # some twenty roundings of 2^-24; bfloat16's 2^-8 on top
    tolerance = 3e-6 + (2 ** -8 if out_dtype == torch.bfloat16 else 0.0)
    assert ((out[:, :heads * dv].double() - want).abs() <= tolerance * want.abs() + 1e-30).all() and (out[:, heads * dv:] == 5.0).all()
