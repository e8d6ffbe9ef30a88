"""The chunked delta rule's scratch per (chunk, head) (no GPU needed)."""
import ctypes

import pytest


@pytest.mark.parametrize("dk,dv,want", [(64, 64, 3 * 64 * 64 // 2 + 2 * 64 * 64 + 4), (1, 1, 7 * 64 * 64 // 2 + 4), (65, 64, 2 * 64 * 64 + 64),
                                        (64, 65, 2 * 64 * 64 + 64), (128, 128, 2 * 64 * 64 + 64), (256, 512, 2 * 64 * 64 + 64)])
def test_each_form_gets_what_it_uses(dk, dv, want):
    """Heads of up to 64 x 64: three planes of N, the states, R and a decay; wider ones: T, P and the decays of a chunk."""
    from cisr_b200.ops import build
    lib = build.load_library("delta.cu")
    lib.cisr_delta_chunk_table_floats.restype = ctypes.c_longlong
    assert lib.cisr_delta_chunk_table_floats(dk, dv) == want
