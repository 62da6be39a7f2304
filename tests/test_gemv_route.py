"""How matvecs of one row are launched on a 148-SM part.  The choice is host code, so this needs no GPU."""
import ctypes

import pytest

import native_build
from litenn_b200 import capi, synth

SMS = 148
X = 1 << 20  # an address; nothing reads it


@pytest.fixture(scope="module")
def lib(qmm_lib):
    return native_build.load("gemv_route", device_code=False, link_library=capi.LIB_PATH)


@pytest.fixture(scope="module")
def one_launch(lib):
    lib.gemv_one_launch.argtypes = [ctypes.c_int] + [ctypes.c_int64] * 2 + [ctypes.c_uint64] * 2 + [ctypes.c_int]
    return lambda fmt, n, k, x, y: bool(lib.gemv_one_launch(fmt, n, k, x, y, SMS))


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("n,k", [(4096, 4096), (1024, 4096), (4096, 1024), (5, 256)])
def test_a_result_over_its_input_is_packed_by_a_kernel_of_its_own(one_launch, fmt, n, k):
    """CTAs of the one launch store y while others read x."""
    assert one_launch(fmt, n, k, X, X + 4 * k) and one_launch(fmt, n, k, X, X - 4 * n)  # side by side
    for y in (X, X + 4, X + 4 * (k - 1), X - 4 * (n - 1), X - 4 * (n // 2), X + 4 * (k // 2)):
        assert not one_launch(fmt, n, k, X, y), y - X


def test_long_rows_of_few_channels_are_read_by_blocks_of_one_row_tile(lib):
    """A packed product groups four row tiles in a block, which leaves most of the chip idle where there are few."""
    lib.swiglu_packs.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    for k, channels in ((8192, 1024), (8192, 1792), (7680, 2048), (5120, 1280), (12288, 1536), (4352, 512)):
        assert not lib.swiglu_packs(channels, k, SMS), (k, channels)
    for k, channels in ((8192, 2304), (8192, 28672), (5120, 3456), (4096, 11008), (4096, 1376), (2048, 512)):
        assert lib.swiglu_packs(channels, k, SMS), (k, channels)
