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


STORE, RESIDUAL, GATE_UP = 0, 1, 3
Q4_0, Q8_0, Q4_K, Q6_K = synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K


@pytest.mark.parametrize("epi,chained,n,k,wave,small", [
    # packed vector on its own: short rows of few tiles per SM stay with small blocks
    (STORE, 0, 16000, 768, (Q8_0, Q6_K), (Q4_0, Q4_K)),
    (STORE, 0, 10777, 1536, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    (STORE, 0, 11008, 2048, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    (STORE, 0, 16384, 2048, (Q4_0, Q8_0, Q4_K, Q6_K), ()),
    (STORE, 0, 4096, 4096, (Q4_0, Q8_0, Q4_K, Q6_K), ()),
    (STORE, 0, 10240, 8192, (Q4_0, Q8_0, Q4_K, Q6_K), ()),
    (STORE, 0, 5000, 6144, (Q6_K,), (Q4_0, Q8_0, Q4_K)),
    (STORE, 0, 36000, 8192, (Q4_K, Q6_K), (Q4_0, Q8_0)),
    # vocabularies
    (STORE, 1, 32000, 4096, (Q4_0, Q4_K, Q6_K), (Q8_0,)),
    (STORE, 1, 12288, 4096, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    # residual matvecs
    (RESIDUAL, 0, 8192, 1024, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    (RESIDUAL, 0, 8192, 4096, (Q6_K,), (Q4_0, Q8_0, Q4_K)),
    (RESIDUAL, 0, 8192, 28672, (Q4_0, Q8_0, Q4_K, Q6_K), ()),
    (RESIDUAL, 0, 12288, 8192, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    (RESIDUAL, 0, 16384, 5120, (Q8_0, Q6_K), (Q4_0, Q4_K)),
    # gate|up
    (GATE_UP, 1, 22016, 2048, (), (Q4_0, Q8_0, Q4_K, Q6_K)),
    (GATE_UP, 1, 22016, 4096, (Q8_0, Q4_K), (Q4_0, Q6_K)),
    (GATE_UP, 1, 28672, 4096, (Q4_0, Q8_0, Q4_K, Q6_K), ()),
    (GATE_UP, 1, 57344, 8192, (Q4_0, Q8_0, Q4_K), (Q6_K,)),
])
def test_one_wave_is_taken_where_it_is_the_faster_form(lib, epi, chained, n, k, wave, small):
    for fmt in wave + small:
        assert bool(lib.gemv_takes_one_wave(fmt, epi, ctypes.c_int64(n), ctypes.c_int64(k), chained, SMS)) == (fmt in wave), fmt


@pytest.mark.parametrize("epi,xf32", [(STORE, 1), (STORE, 0), (RESIDUAL, 0), (GATE_UP, 0)])
@pytest.mark.parametrize("fmt", [Q4_0, Q8_0, Q4_K, Q6_K])
def test_every_shape_has_a_form_that_fits_and_every_compiled_form_a_shape(lib, fmt, epi, xf32):
    assert lib.gemv_wave_forms_unreached(fmt, epi, xf32, SMS) == 0
    assert lib.gemv_wave_forms_unreached(fmt, epi, xf32, 74) >= 0  # a part of the chip: the rules scale with it
