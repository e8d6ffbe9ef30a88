"""The quotient of the gates (csrc/common.cuh) against the division operator, bit for bit."""
import ctypes
import subprocess

import pytest
import torch

from cisr_b200.ops import build

pytestmark = pytest.mark.gpu
SOURCE = """
#include "common.cuh"
__global__ void quotients(const float* n, const float* d, float* out, long long count) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = quotient(n[i], d[i]);
}
CISR_EXPORT int run(const float* n, const float* d, float* out, long long count, void* stream) {
    quotients<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, d, out, count);
    return launch_status();
}
"""


@pytest.fixture(scope="module")
def quotient(tmp_path_factory):
    folder = tmp_path_factory.mktemp("quotient")
    (folder / "quotient.cu").write_text(SOURCE)
    subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, *build.BASE_FLAGS, "-I", str(build.CSRC), "-o", str(folder / "quotient.so"), str(folder / "quotient.cu")], check=True)
    lib = ctypes.CDLL(str(folder / "quotient.so"))
    lib.run.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_longlong, ctypes.c_void_p]

    def call(n, d):
        assert n.shape == d.shape and n.dtype == d.dtype == torch.float32 and n.is_contiguous() and d.is_contiguous()
        out = torch.empty_like(n)
        assert lib.run(n.data_ptr(), d.data_ptr(), out.data_ptr(), n.numel(), torch.cuda.current_stream().cuda_stream) == 0
        return out
    return call


def differ(got, want):
    """Elements whose bits differ (any NaN is as good as another)."""
    return (got.view(torch.int32) != want.view(torch.int32)) & ~(got.isnan() & want.isnan())


@pytest.mark.parametrize("slope", [1.0, 1.702])           # of the logistic function: silu, and the clamped gate
@pytest.mark.parametrize("numerator", ["gate", "one"])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_gates(quotient, slope, numerator, sign):
    g = torch.Generator(device="cuda").manual_seed(int(10 * slope))
    for _ in range(2):                                     # sizes even over their logarithm, from 1e-9 to 88
        z = sign * torch.empty(1 << 25, device="cuda").uniform_(-20.723, 4.4773, generator=g).exp_()
        d = 1.0 + torch.exp(-slope * z)
        n = z if numerator == "gate" else torch.ones_like(z)
        assert int(differ(quotient(n, d), n / d).sum()) == 0


def test_ends_of_the_range(quotient):
    inf, nan, most, least = float("inf"), float("nan"), 3.4028234663852886e38, 2.0 ** -149
    # what the gates meet there: tiny numerators over 2, ordinary ones over denominators up to infinity
    tiny = torch.cat((torch.arange(0, 4096) * least, torch.arange(1, 4096) * 2.0 ** -126 / 1024, torch.tensor([2.0 ** -124, 2.0 ** -100, 1e-30])))
    large = torch.cat((torch.tensor([1.0, 2.0, 2.0 ** 100, 2.0 ** 126, 2.0 ** 127, most, inf, nan]), torch.logspace(28, 38.5, 4096),
                       2.0 ** 100 * (1 + torch.arange(-64, 65) * 2.0 ** -23)))
    pairs = [(s * tiny, torch.full_like(tiny, 2.0)) for s in (1.0, -1.0)]
    pairs += [(torch.full_like(large, n), large) for n in (0.0, -0.0, 1.0, -1.0, -64.0, -88.0, -709.0, 2.0 ** -126, -1e-38, inf, -inf, nan)]
    n, d = (torch.cat([p[i] for p in pairs]).float().contiguous() for i in (0, 1))
    got, want = quotient(n.cuda(), d.cuda()).cpu(), n / d
    odd = differ(got, want).nonzero().flatten()
    assert not odd.numel(), [(float(n[i]), float(d[i]), float(got[i]), float(want[i])) for i in odd[:8]]
