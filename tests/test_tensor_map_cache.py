"""The cache of tensor maps, built into a host program with an encoder that writes down what it is asked for (no GPU needed)."""
import subprocess

import pytest

from cisr_b200.ops import build

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#include "tma.cuh"

// a "map" that holds its arguments: base, rank, the boxes
CUresult write_down(CUtensorMap* map, CUtensorMapDataType, cuuint32_t rank, void* base, const cuuint64_t* dims, const cuuint64_t*, const cuuint32_t* box,
                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    unsigned long long words[16] = {(unsigned long long)base, rank};
    for (unsigned i = 0; i < rank; ++i) { words[2 + i] = box[i]; words[8 + i] = dims[i]; }
    memcpy(map, words, sizeof(words));
    return CUDA_SUCCESS;
}
unsigned long long word(const CUtensorMap& map, int i) { unsigned long long words[16]; memcpy(words, &map, sizeof(words)); return words[i]; }

int boxes() {
    CUtensorMap one, two;
    const int status = cached_map(&one, (void*)4096, 512, 256, 64, 128, 2, 1) | cached_map(&two, (void*)4096, 512, 256, 64, 128, 2, 2);
    return status || word(one, 4) != 1 || word(two, 4) != 2;
}
int threads() {
    g_map_cache_limit = 7;                       // emptied again and again
    std::vector<std::thread> all;
    std::vector<int> wrong(8);
    for (int t = 0; t < 8; ++t)
        all.emplace_back([&, t] {
            for (int i = 0; i < 200000; ++i) {
                const long long rows = 128 * (1 + (i * 7 + t) % 13);
                CUtensorMap map;
                if (cached_map(&map, (void*)(4096 * rows), rows, 64, 64) || word(map, 0) != 4096ull * rows || word(map, 9) != (unsigned long long)rows) ++wrong[t];
            }
        });
    for (auto& t : all) t.join();
    int sum = 0;
    for (int w : wrong) sum += w;
    return sum;
}
int main(int, char** argv) {
    g_encode = write_down;
    return (argv[1][0] == 'b' ? boxes() : threads()) != 0;
}
"""


@pytest.mark.parametrize("part", ["boxes", "threads"])        # boxes of another size are told apart; threads share the cache
def test_cache(part, tmp_path):
    (tmp_path / "maps.cu").write_text(PROGRAM)
    made = subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC), "-o", str(tmp_path / "maps"),
                           str(tmp_path / "maps.cu")], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    assert subprocess.run([tmp_path / "maps", part], timeout=120).returncode == 0
