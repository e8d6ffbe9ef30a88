"""The chunked recurrences whose products run as split bfloat16 parts on the tensor cores, at sizes around their 64 x 64
tiles, against the recurrence token by token in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
# 64 terms per product with four roundings, a few products and exponentials per result: some 2^-24 each, 4e-7 in all
BOUND = 4e-7


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device="cuda")


def step_lists(lens):
    req, t0, first = [], [], []
    for r, n in enumerate(lens):
        first.append(len(req))
        for t in range(0, n, 64):
            req.append(r); t0.append(t)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    return starts, (i32(req), i32(t0), i32(first), len(req))


def error(got, want):
    assert torch.isfinite(got).all()
    return float((got.double() - want).norm() / want.norm())


SIZES = [(64, 64, [64]), (128, 128, [65, 127]), (50, 37, [64, 130]), (72, 50, [191]), (4, 4, [64, 200]), (130, 66, [128, 129])]


@pytest.mark.parametrize("dk,dv,lens", SIZES)
def test_lightning_chunks(dk, dv, lens):
    from cisr_b200.ops import kernels
    heads, g = 3, torch.Generator(device="cuda").manual_seed(dk + dv)
    starts, chunks = step_lists(lens)
    proj = torch.randn(sum(lens), heads * (2 * dk + dv), generator=g, device="cuda")
    decay = torch.tensor([0.96, 0.998, 1.0], device="cuda")
    state = torch.randn(len(lens), heads * dk * dv, generator=g, device="cuda")
    silu = lambda x: x * torch.sigmoid(x)
    q, k, v = (silu(x) for x in proj.double().split([heads * dk, heads * dk, heads * dv], 1))
    want, ends = [], []
    for r, n in enumerate(lens):
        S = state[r].double().view(heads, dv, dk).transpose(1, 2).clone()
        for t in range(starts[r], starts[r] + n):
            S = decay.double()[:, None, None] * S + k[t].view(heads, dk, 1) * v[t].view(heads, 1, dv)
            want.append(torch.einsum("hkv,hk->hv", S, q[t].view(heads, dk)).reshape(-1))
        ends.append(S.transpose(1, 2).reshape(-1))
    o = torch.full((sum(lens), heads * dv), float("nan"), device="cuda")
    kernels.lightning_recurrence(proj, 0, heads * dk, 2 * heads * dk, decay, state, i32(range(len(lens))), i32(starts), i32(lens), len(lens), o, heads, dk, dv,
                                 least=64, chunks=chunks)
    assert error(o, torch.stack(want)) < BOUND and error(state, torch.stack(ends)) < BOUND


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("N,dv,lens", SIZES)
def test_gated_chunks(N, dv, lens, norm):
    from cisr_b200.ops import kernels
    heads, groups, g = 4, 2, torch.Generator(device="cuda").manual_seed(N + dv)
    starts, chunks = step_lists(lens)
    T = sum(lens)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k, v = rand(T, groups * N), rand(T, groups * N), rand(T, heads * dv)
    la, gain = -3.0 * torch.rand(T, heads, generator=g, device="cuda") ** 6, torch.rand(T, heads, generator=g, device="cuda")
    state = rand(len(lens), heads * N * (dv + int(norm)))
    y, yn = torch.full((T, heads, dv), float("nan"), device="cuda"), torch.full((T, heads), float("nan"), device="cuda") if norm else None
    Q, K = (x.double().view(T, groups, N).repeat_interleave(2, 1) for x in (q, k))
    V = v.double().view(T, heads, dv)
    want, want_n, ends = [], [], []
    for r, n in enumerate(lens):
        S = state[r, :heads * N * dv].double().view(heads, N, dv).clone()
        m = state[r, heads * N * dv:].double().view(heads, N).clone() if norm else torch.zeros(heads, N, device="cuda", dtype=torch.float64)
        for t in range(starts[r], starts[r] + n):
            e, gk = la[t].double().exp(), gain[t].double()[:, None] * K[t]
            S, m = e[:, None, None] * S + gk[:, :, None] * V[t][:, None], e[:, None] * m + gk
            want.append(0.5 * torch.einsum("hkv,hk->hv", S, Q[t]))
            want_n.append(0.5 * (m * Q[t]).sum(-1))
        ends.append(torch.cat([S.reshape(-1)] + ([m.reshape(-1)] if norm else [])))
    kernels.gated_recurrence(q, 0, k, 0, v, 0, la, gain, state, i32(range(len(lens))), i32(starts), i32(lens), len(lens), y, groups, N, q_scale=0.5, yn=yn,
                             least=64, chunks=chunks)
    assert error(y, torch.stack(want)) < BOUND and error(state, torch.stack(ends)) < BOUND
    if norm:
        assert error(yn, torch.stack(want_n)) < BOUND


@pytest.mark.parametrize("dk,dv,heads,kvh,lens", [(64, 64, 4, 1, [64, 65, 200]), (48, 40, 2, 1, [127, 128]), (33, 7, 3, 3, [129]), (16, 16, 2, 2, [64]), (64, 1, 1, 1, [191])])
def test_delta_forms(dk, dv, heads, kvh, lens):
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    starts, (req, t0, first, n_chunks) = step_lists(lens)
    T = sum(lens)
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, kvh, dk, generator=g, device="cuda"), dim=-1)
    q, k, v = unit() * dk ** -0.5, unit(), torch.randn(T, heads, dv, generator=g, device="cuda")
    qkv = torch.cat([x.reshape(T, -1) for x in (q, k, v)], dim=1).contiguous()
    beta = torch.rand(T, heads, generator=g, device="cuda")
    decay = torch.exp(-3.0 * torch.rand(T, heads, generator=g, device="cuda") ** 6)
    state = torch.randn(len(lens), heads * dk * dv, generator=g, device="cuda")
    Q, K = (x.double().repeat_interleave(heads // kvh, 1) for x in (q, k))
    want, ends = [], []
    for r, n in enumerate(lens):
        S = state[r].double().view(heads, dk, dv).clone()
        for t in range(starts[r], starts[r] + n):
            S = decay[t].double()[:, None, None] * S
            u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hkv,hk->hv", S, K[t]))
            S = S + K[t][:, :, None] * u[:, None]
            want.append(torch.einsum("hkv,hk->hv", S, Q[t]))
        ends.append(S.reshape(-1))
    o = torch.full((T, heads, dv), float("nan"), device="cuda")
    kernels.delta_chunks(qkv, beta, decay, req, t0, n_chunks, first, state, i32(range(len(lens))), i32(starts), i32(lens), o, len(lens), heads, kvh, dk, dv, 64)
    assert error(o, torch.stack(want)) < BOUND and error(state, torch.stack(ends)) < BOUND


def lightning_case(lens, dk, dv, heads, decay, change):
    """The chunked recurrence and the token-by-token one in float64 (silu in float, as the kernel takes it) for operands that
    `change` has altered: outputs and states of both."""
    from cisr_b200.ops import kernels
    g = torch.Generator(device="cuda").manual_seed(dk + dv)
    starts, chunks = step_lists(lens)
    proj = torch.randn(sum(lens), heads * (2 * dk + dv), generator=g, device="cuda")
    state = torch.randn(len(lens), heads * dk * dv, generator=g, device="cuda")
    change(proj, state)
    q, k, v = (torch.nn.functional.silu(x).double() for x in proj.split([heads * dk, heads * dk, heads * dv], 1))
    want, ends = [], []
    for r, n in enumerate(lens):
        S = state[r].double().view(heads, dv, dk).transpose(1, 2).clone()
        for t in range(starts[r], starts[r] + n):
            S = decay.double()[:, None, None] * S + k[t].view(heads, dk, 1) * v[t].view(heads, 1, dv)
            want.append(torch.einsum("hkv,hk->hv", S, q[t].view(heads, dk)).reshape(-1))
        ends.append(S.transpose(1, 2).reshape(-1))
    o = torch.full((sum(lens), heads * dv), float("nan"), device="cuda")
    kernels.lightning_recurrence(proj, 0, heads * dk, 2 * heads * dk, decay, state, i32(range(len(lens))), i32(starts), i32(lens), len(lens), o, heads, dk, dv,
                                 least=64, chunks=chunks)
    return (o, state), (torch.stack(want), torch.stack(ends))


def same_where_finite(got, want):
    ok = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), ok)
    assert float((got.double() - want)[ok].norm() / want[ok].norm()) < BOUND


@pytest.mark.parametrize("odd", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 13, 30, 63, 100, 150])
def test_lightning_non_finite_values_reach_later_tokens_only(at, odd):
    heads, dk, dv = 2, 72, 50

    def change(proj, state):
        proj[at, 2 * heads * dk + 3] = odd                           # v of head 0, column 3
        proj[at + 20, 2 * heads * dk + dv + 7] = float("nan")        # v of head 1, column 7
        proj[170, 5] = float("nan")                                  # q of head 0: token 170 alone
    for got, want in zip(*lightning_case([191], dk, dv, heads, torch.tensor([0.9, 1.0], device="cuda"), change)):
        same_where_finite(got, want)


def test_lightning_floats_beyond_the_largest_bfloat16():
    def change(proj, state):
        proj[:, :2 * 2 * 16] *= 0.05
        proj[20, 2 * 2 * 16 + 1] = 3.4e38
        state[0, :16] = -3.4e38
    for got, want in zip(*lightning_case([130], 16, 16, 2, torch.tensor([0.5, 0.9], device="cuda"), change)):
        same_where_finite(got, want)


@pytest.mark.parametrize("at", [0, 13, 37, 70])
def test_delta_non_finite_values_reach_later_tokens_only(at):
    from cisr_b200.ops import kernels
    dk, dv, heads, T = 48, 40, 2, 130
    g = torch.Generator(device="cuda").manual_seed(at)
    starts, (req, t0, first, n_chunks) = step_lists([T])
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, heads, dk, generator=g, device="cuda"), dim=-1)
    q, k, v = unit() * dk ** -0.5, unit(), torch.randn(T, heads, dv, generator=g, device="cuda")
    v[at, 0, 3] = float("inf")                 # head 0: one value
    k[at, 1] = float("nan")                    # head 1: a whole key
    qkv = torch.cat([x.reshape(T, -1) for x in (q, k, v)], dim=1).contiguous()
    beta, decay = torch.rand(T, heads, generator=g, device="cuda"), 1 - 0.1 * torch.rand(T, heads, generator=g, device="cuda")
    state = torch.randn(1, heads * dk * dv, generator=g, device="cuda")
    S, want = state[0].double().view(heads, dk, dv).clone(), []
    for t in range(T):
        S = decay[t].double()[:, None, None] * S
        u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hkv,hk->hv", S, k[t].double()))
        S = S + k[t].double()[:, :, None] * u[:, None]
        want.append(torch.einsum("hkv,hk->hv", S, q[t].double()))
    o = torch.full((T, heads, dv), float("nan"), device="cuda")
    kernels.delta_chunks(qkv, beta, decay, req, t0, n_chunks, first, state, i32([0]), i32(starts), i32([T]), o, 1, heads, heads, dk, dv, 64)
    same_where_finite(o, torch.stack(want))
    same_where_finite(state, S.reshape(1, -1))


def test_lightning_decay_of_zero():
    """Each token alone: o = (q . k) v, also where a decay is too small for a float."""
    for got, want in zip(*lightning_case([64, 130], 40, 24, 3, torch.tensor([0.0, 1e-46, 0.9], device="cuda"), lambda proj, state: None)):
        same_where_finite(got, want)
