"""The key and value rings of the tcgen05 prompt attention: no wait on a slot's barrier may skip a phase of it.

A wait on an mbarrier looks at one bit of its phase, so a warp that waits for turn t of a slot must have waited for every
earlier turn of it: after a skipped turn the wait can pass one phase early, before the tile has landed.  The test walks the
tiles as the product warps do, with the ring sizes that the built library reports (no GPU needed)."""
import pytest


def rings(dim):
    from cisr_b200.ops import build
    return build.load_library("attention_tcgen05.cu", {"HEAD_DIM": dim})


def waits(warps, shared, n_tiles):
    """Per product warp the tiles it waits for, in order."""
    order = [j for j in range(n_tiles)]
    if warps == 1:
        return [order]                                       # one warp takes the streams in turn: every tile, in order
    return [order[0::2], order[1::2]] if shared else [order, order]


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("values", [False, True])
@pytest.mark.parametrize("dim", [64, 128])
def test_every_turn_of_a_slot_is_waited_for(dim, values, shared):
    lib = rings(dim)
    slots, warps = lib.cisr_attn_tcgen05_slots(int(values), int(shared)), lib.cisr_attn_tcgen05_product_warps()
    for tiles in waits(warps, shared, 97):
        seen = {}
        for j in tiles:
            slot, turn = j % slots, j // slots
            assert turn == seen.get(slot, -1) + 1, f"tile {j}: turn {turn} of slot {slot} after turn {seen.get(slot)}"
            seen[slot] = turn
