"""How a matvec of one fp32 vector is launched on a 148-SM part.  The choice is host code, so this needs no GPU."""
import ctypes

import pytest

import native_build
from litenn_b200 import capi, synth

SMS = 148
X = 1 << 20  # an address; nothing reads it


@pytest.fixture(scope="module")
def one_launch(qmm_lib):
    lib = native_build.load("gemv_route", device_code=False, link_library=capi.LIB_PATH)
    lib.gemv_one_launch.argtypes = [ctypes.c_int] + [ctypes.c_int64] * 2 + [ctypes.c_uint64] * 2 + [ctypes.c_int]
    return lambda fmt, n, k, x, y: bool(lib.gemv_one_launch(fmt, n, k, x, y, SMS))


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("n,k", [(4096, 4096), (1024, 4096), (4096, 1024), (5, 256)])
def test_a_result_over_its_input_is_packed_by_a_kernel_of_its_own(one_launch, fmt, n, k):
    """CTAs of the one launch store y while others read x."""
    assert one_launch(fmt, n, k, X, X + 4 * k) and one_launch(fmt, n, k, X, X - 4 * n)  # side by side
    for y in (X, X + 4, X + 4 * (k - 1), X - 4 * (n - 1), X - 4 * (n // 2), X + 4 * (k // 2)):
        assert not one_launch(fmt, n, k, X, y), y - X
