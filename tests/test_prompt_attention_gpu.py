"""The tcgen05 prompt attention with tiles of 256 and of 128 queries, at the edges of its tiles, against plain softmax."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
PAGE = 16


def plain(q, k, v, window, keep_first, sink, cap):
    """q at the last positions of k, v [S, heads, D], in float64."""
    n, hq, d = q.shape
    s_len, hkv = k.shape[:2]
    qpos, kpos = torch.arange(s_len - n, s_len)[:, None], torch.arange(s_len)[None]
    hidden = kpos > qpos
    if window:
        hidden |= (kpos <= qpos - window) & (kpos >= keep_first)
    out = torch.empty(n, hq, d, dtype=torch.float64)
    for h in range(hq):
        g = h // (hq // hkv)
        s = q[:, h] @ k[:, g].T * d ** -0.5
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat((s, torch.full((n, 1), sink, dtype=torch.float64)), dim=1)
        p = torch.softmax(s, dim=-1)
        out[:, h] = p[:, :s_len] @ v[:, g]
    return out


def run(portions, d, hq, hkv, span, window=0, keep_first=0, sink=None, cap=None, sharp=1.0, spoiled=None):
    """portions: (queries, keys before them) per request; cache rows that no request wrote hold NaN, and so does the first
    request's key `spoiled`."""
    from cisr_b200.ops import kernels
    g = torch.Generator().manual_seed(7 + d + len(portions))
    pages = sum(-(-(n + b) // PAGE) for n, b in portions) + 2
    k_cache = torch.full((pages, hkv, PAGE, d), float("nan"), dtype=torch.bfloat16)
    v_cache = torch.full_like(k_cache, float("nan"))
    order = torch.randperm(pages, generator=g).tolist()
    table = np.full((len(portions), 64), -1, dtype=np.int32)
    qs, want = [], []
    for r, (n, before) in enumerate(portions):
        total = n + before
        q = (torch.randn(n, hq, d, generator=g) * sharp).bfloat16()
        k, v = (torch.randn(total, hkv, d, generator=g).bfloat16() for _ in range(2))
        for i in range(-(-total // PAGE)):
            page = order.pop()
            table[r, i] = page
            rows = min(PAGE, total - i * PAGE)
            k_cache[page, :, :rows] = k[i * PAGE:i * PAGE + rows].transpose(0, 1)
            v_cache[page, :, :rows] = v[i * PAGE:i * PAGE + rows].transpose(0, 1)
        if spoiled is not None and r == 0:
            for cache in (k_cache, v_cache):
                cache[table[0, spoiled // PAGE], :, spoiled % PAGE] = float("nan")
        qs.append(q)
        want.append(plain(q.double(), k.double(), v.double(), window, keep_first, sink, cap))
    dev = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32), device="cuda")
    q = torch.cat(qs).cuda()
    out = torch.full_like(q, float("nan"))
    lens = [n for n, _ in portions]
    tiles = [(r, q0) for r, n in enumerate(lens) for q0 in reversed(range(0, n, span))]
    kernels.attn_prefill_wide(q, out, k_cache.cuda(), v_cache.cuda(), dev(range(len(lens))), dev(table), dev([t[0] for t in tiles]), dev([t[1] for t in tiles]),
                              dev(np.cumsum([0] + lens[:-1])), dev(lens), dev([n + b for n, b in portions]), hq, hkv, PAGE, d ** -0.5, window,
                              sink=sink, keep_first=keep_first, softcap=cap, span=span)
    kernels.raise_if_kernel_gave_up()
    return out.double().cpu(), torch.cat(want)


def check(out, want):
    """P and the result are rounded to bfloat16 (2^-9 each, relative to the row's largest terms): 2e-2 of the values' scale."""
    assert torch.isfinite(out).all()
    assert float((out - want).norm() / want.norm()) < 6e-3
    assert float((out - want).abs().max()) < 2e-2 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("span", [128, 256])
@pytest.mark.parametrize("d,hq,hkv", [(64, 3, 1), (128, 2, 2)])
def test_edges_of_the_tiles(d, hq, hkv, span):
    check(*run([(2, 0), (127, 1), (128, 0), (129, 127), (256, 0), (257, 130), (300, 511)], d, hq, hkv, span))


@pytest.mark.parametrize("span", [128, 256])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window,keep_first", [(1, 0), (100, 0), (128, 5), (200, 130), (2000, 3)])
def test_windows_and_kept_keys(d, window, keep_first, span):
    check(*run([(200, 300), (259, 420), (5, 700)], d, 2, 1, span, window=window, keep_first=keep_first, sink=0.3))


@pytest.mark.parametrize("span", [128, 256])
@pytest.mark.parametrize("cap", [20.0, 80.0])       # with and without a running max
def test_bent_scores(cap, span):
    check(*run([(140, 0), (256, 77)], 64, 2, 1, span, cap=cap, sharp=4.0))


@pytest.mark.parametrize("span", [128, 256])
@pytest.mark.parametrize("d", [64, 128])
def test_a_max_that_moves_rescales_the_rows_before_it(d, span):
    check(*run([(256, 512), (90, 900)], d, 2, 2, span, sharp=12.0))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("keep_first", [0, 5, 128, 150, 300])
@pytest.mark.parametrize("n,before,window", [(256, 300, 128), (200, 300, 100), (512, 40, 128), (300, 700, 257), (256, 127, 128), (256, 128, 130)])
def test_windows_of_both_streams(d, keep_first, n, before, window):
    check(*run([(n, before)], d, 2, 1, 256, window=window, keep_first=keep_first))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("key", [173, 200, 255])
def test_a_key_before_the_second_streams_window_does_not_reach_it(d, key):
    """Queries 428 to 555 see keys from 301 on; the tile of keys 128 to 255 belongs to the queries before them."""
    out, want = run([(256, 300)], d, 2, 1, 256, window=128, spoiled=key)
    check(out[128:], want[128:])
