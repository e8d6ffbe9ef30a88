"""Which tcgen05 kernel a plain product goes to, by its sizes, the device's SMs and the switch (no GPU needed)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def choices(sizes, sms, **env):
    code = ("from cisr_b200.ops import build; lib = build.load_library('gemm_tcgen05.cu');"
            f"print(*(lib.cisr_gemm_tcgen05_plain_choice(m, n, k, {sms}) for m, n, k in {sizes}))")
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True, check=True).stdout
    return [int(x) for x in out.split()]


SIZES = [(2048, 64, 4096), (128, 33, 2048), (9472, 64, 2048), (9473, 64, 2048), (2048, 64, 2040), (200, 576, 1536), (64, 4096, 4096), (256, 18944, 520),
         (2048, 28672, 4096)]


@pytest.mark.parametrize("sms,want", [(148, [6412, 6412, 6412, 0, 0, 6412, 12814, 25611, 0]), (132, [6412, 6412, 0, 0, 0, 6412, 12814, 25621, 0])])
def test_choice_by_sizes(sms, want):
    assert choices(SIZES, sms) == want


def test_the_switch_sends_every_product_to_the_persistent_kernel():
    assert choices(SIZES, 148, CISR_GEMM_DEEP="0") == [0] * len(SIZES)
