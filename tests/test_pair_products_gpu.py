"""The tcgen05 products on pairs of SMs: every tile width, edges of the 256-row tiles, one round and more, short and ragged K."""
import pytest
import torch

SIZES = [(257, 9000, 1096), (1400, 5184, 1096), (600, 9000, 264), (1400, 4000, 1032), (2533, 2052, 1032), (300, 37001, 72), (2049, 5184, 136), (511, 22222, 200), (4000, 700, 1096)]
GATED = [(1000, 2052, 1096), (2049, 5184, 1096), (2049, 5184, 136), (1000, 4804, 1096), (513, 9001, 136), (2533, 700, 1096), (2100, 2056, 72), (300, 8192, 1096), (1281, 3000, 264)]
ROTATED = [(700, 64, 16, 64, 264), (2533, 32, 32, 64, 136), (1500, 32, 8, 128, 72), (300, 66, 40, 128, 1096), (520, 64, 64, 64, 1096)]


def test_sizes_reach_every_width():
    """No GPU needed: the tests below cover the widths the rule chooses from."""
    from cisr_b200.ops import build
    lib = build.load_library("gemm_tcgen05.cu")
    width = lib.cisr_gemm_tcgen05_pair_width
    assert all(lib.cisr_gemm_tcgen05_plain_choice(m, n, k, 148) == 0 for m, n, k in SIZES)
    assert {width(m, n, k, 0, 0, 148) for m, n, k in SIZES} | {width(m, n, k, 1, 0, 148) for m, n, k in GATED} == {256, 224, 192, 160, 128}
    assert {width(m, (q + 2 * kv) * d, k, 0, d, 148) for m, q, kv, d, k in ROTATED if d == 64} <= {256, 192, 128}
    assert {width(m, (q + 2 * kv) * d, k, 0, d, 148) for m, q, kv, d, k in ROTATED if d == 128} <= {256, 128}


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,kk", SIZES)
@pytest.mark.parametrize("accumulate", [False, True])
def test_plain(m, n, kk, accumulate):
    from test_few_tiles_gpu import test_plain as plain
    plain(m, n, kk, accumulate)


@pytest.mark.gpu
@pytest.mark.parametrize("m,inter,kk", GATED)
@pytest.mark.parametrize("gate", ["silu", "gelu_tanh", "gated_clamp"])
def test_gated(m, inter, kk, gate):
    from test_few_tiles_gpu import test_gated as gated
    gated(m, inter, kk, gate)


@pytest.mark.gpu
@pytest.mark.parametrize("m,hq,hkv,dim,kk", ROTATED)
def test_rotated(m, hq, hkv, dim, kk):
    from test_few_tiles_gpu import test_rotated as rotated
    rotated(m, hq, hkv, dim, kk)
