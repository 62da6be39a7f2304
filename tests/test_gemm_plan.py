"""Which form of the prefill GEMM a product takes on a 148-SM part.  The choice is host code, so this needs no GPU: it holds
the labels of the forms test to the forms, and every plan of the declared range to what the kernels accept."""
import ctypes
import itertools

import pytest

import native_build
from litenn_b200 import capi, synth
from test_gpu_gemm_forms import CASES

SMS = 148


@pytest.fixture(scope="module")
def plan(qmm_lib):
    lib = native_build.load("gemm_forms", device_code=False, link_library=capi.LIB_PATH)
    lib.gemm_plan_of.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int] * 2 + [ctypes.c_void_p]

    def of(n, k, m, keep_order=False):
        out = (ctypes.c_int * 5)()
        lib.gemm_plan_of(n, k, m, SMS, int(keep_order), out)
        return dict(zip(("nb", "tokens", "t_tiles", "splits", "groups"), out))
    return of


EXPECTED = {
    "one CTA per tile": lambda p: p["nb"] == 1 and p["splits"] == 1,
    "split": lambda p: p["nb"] == 1 and p["splits"] > 1,
    "split, several token tiles": lambda p: p["nb"] == 1 and p["splits"] > 1 and p["t_tiles"] > 1,
    "two blocks": lambda p: p["nb"] == 2,
    "shared memory": lambda p: p["groups"] > 0,
}


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q4_K])
@pytest.mark.parametrize("form,m,n,k", CASES)
def test_the_forms_test_reaches_the_forms_it_names(plan, form, m, n, k, fmt):
    unit = synth.BLOCK_ELEMS[fmt]
    assert EXPECTED[form](plan(n, (k + unit - 1) // unit * unit, m))


def test_every_plan_is_one_the_kernels_accept(plan):
    for n, k, m in itertools.product((3, 130, 512, 4096, 28672), (32, 288, 4096, 28672),
                                     (1, 16, 17, 127, 128, 129, 256, 257, 700, 2048)):
        p = plan(n, k, m)
        row_tiles = (n + 15) // 16
        if p["groups"]:
            assert p["groups"] <= row_tiles <= 16 * p["groups"]
        else:
            assert p["tokens"] % 16 == 0 and 16 <= p["tokens"] <= 128
            assert (p["t_tiles"] - 1) * p["tokens"] < m <= p["t_tiles"] * p["tokens"]
            assert p["splits"] in ((1, 2, 4, 8) if p["nb"] == 1 else (1,)) and p["splits"] <= (k + 255) // 256
        assert plan(n, k, m, keep_order=True)["groups"] > 0
