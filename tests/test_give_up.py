"""Kernels that give up: what they wait for before they free their tensor memory and leave (no GPU needed; no wait is made to run out on one)."""
import re
import subprocess

from cisr_b200.ops import build

PROGRAM = r"""
#include "tcgen05.cuh"

// the blocks that may still be on their way are the last one of each stage: which stage, and the parity of the turn that it is on
int main() {
    for (int stages = 1; stages <= 8; ++stages)
        for (int requested = 0; requested < 40; ++requested) {
            int last[8], turns[8] = {};
            for (int s = 0; s < stages; ++s) last[s] = -1;
            for (int j = 0; j < requested; ++j) last[j % stages] = j, ++turns[j % stages];
            int seen = 0;
            for (int j = first_in_flight(requested, stages); j < requested; ++j, ++seen) {
                const BlockAt at(j, stages);
                if (last[at.stage] != j || at.turn != (unsigned)(turns[at.stage] - 1) % 2) return 1;
            }
            if (seen != (requested < stages ? requested : stages)) return 2;
        }
    return 0;
}
"""


def test_blocks_in_flight(tmp_path):
    (tmp_path / "ring.cu").write_text(PROGRAM)
    made = subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC), "-o", str(tmp_path / "ring"),
                           str(tmp_path / "ring.cu")], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    assert subprocess.run([tmp_path / "ring"]).returncode == 0


def test_products_and_copies_are_waited_for_before_tensor_memory_is_freed():
    """In the text of every kernel with products on tcgen05, between its last role and the instruction that frees its tensor memory."""
    kernels = 0
    for name in ("gemm_tcgen05.cu", "gemm_float.cu", "few_gemm.cu", "attention_tcgen05.cu"):
        text = (build.CSRC / name).read_text()
        shared = "meet_pair(" in text and re.search(r"void meet_pair\(.*?\n}\n", text, re.DOTALL).group(0)
        for part in text.split("__global__")[1:]:
            if "tcgen05.dealloc" not in part:
                continue
            kernels += 1
            end = part[:part.index("tcgen05.dealloc")][-900:]
            end = end + shared if "meet_pair(" in end else end
            assert "wait_for_products" in end, (name, part[:120])
            assert "wait_for_copies" in end or "cp.async.bulk" not in part and "tma_load" not in part, (name, part[:120])
    assert kernels == 7
