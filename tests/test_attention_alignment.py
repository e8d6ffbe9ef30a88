"""Attention reads queries, keys and values by 16 bytes: buffers that do not start there are refused, never launched on (no GPU needed)."""
import pytest

from cisr_b200.ops import build

LIBRARIES = [("attention_float.cu", {"HEAD_DIM": 16}), ("attention.cu", {"HEAD_DIM": 16, "STORAGE_BF16": 0}), ("attention.cu", {"HEAD_DIM": 16, "STORAGE_BF16": 1}),
             ("attention_mma.cu", {"HEAD_DIM": 16})]


@pytest.mark.parametrize("source,defines", LIBRARIES)
@pytest.mark.parametrize("field", [0, 2, 3])             # q, k_cache, v_cache
def test_entries_refuse_what_they_cannot_read(source, defines, field):
    lib = build.load_library(source, defines)
    at = [1 << 40] * 4
    at[field] += 4
    prefill = lib.cisr_attn_prefill_float if source == "attention_float.cu" else lib.cisr_attn_prefill
    assert prefill(*at, 0, 0, 1, 0, 0, 1, 0, 0, 0, 2, 1, 16, 0.25, 0.0, 0, 0, 0.0, 0, 0) == -2
    if source != "attention_float.cu":
        merge = (1,) if source == "attention_mma.cu" else ()
        assert lib.cisr_attn_decode(*at, 0, 0, 1, 0, 1, 0, 0, 0, 0, 2, 1, 16, 0.25, 0.0, 0, 0, 64, 1, *merge, 0.0, 0, 0) == -2
