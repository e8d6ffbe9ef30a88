"""The packed arguments of the weight-streaming products (no GPU needed)."""
import pytest

from cisr_b200.ops import kernels


@pytest.mark.parametrize("at,value", [(19, None), (22, 2 ** 31), (25, -2 ** 31 - 1), (30, "8"), (0, None)])
def test_what_does_not_fit_is_refused_as_every_wrong_argument_is(at, value):
    values = [0] * 19 + [0.0] * 3 + [0] * 15
    assert len(kernels._skinny_call(*values)) == 19 * 8 + 3 * 8 + 15 * 4
    values[at] = value
    with pytest.raises(kernels.KernelError, match="skinny_gemm"):
        kernels._skinny_call(*values)
