"""The order of dependency waits and releases inside kernels that launch while the kernel before them still runs.

A broken order is a race that a run rarely shows, so this reads the kernels' source.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "litenn_b200", "csrc")


def kernel_body(file, name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    start = text.index("{", re.search(r"\b%s\(" % name, text).start())
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]


@pytest.mark.parametrize("name", ["embed_row_kernel", "embed_pack_kernel"])
def test_the_first_kernel_of_a_step_waits_before_it_releases_the_next(name):
    """attn_fused_kernel reads the position and the cached keys ahead of its own wait: the step before has to be over."""
    body = kernel_body("llama_kernels.cu", name)
    assert body.index("pdl_sync()") < body.index("pdl_trigger()")
    assert body.count("pdl_trigger()") == 1


@pytest.mark.parametrize("file,name", [("qmm_gemm.cu", "gemm_ts_kernel"), ("qmm_gemm_smem.cu", "gemm_tcgen05_kernel")])
def test_every_warp_of_a_gemm_waits_for_the_kernel_before_ahead_of_a_bounded_wait(file, name):
    """A limit that ran while an earlier kernel still works would fail a healthy product."""
    body = kernel_body(file, name)
    roles = re.split(r"\bif \(warp == |\} else if \(warp == |\} else \{\n(?=\s+const int (?:quad|dw) )", body)
    waiting = [r for r in roles if re.search(r"g_mbar_(?:wait|poll)", r)]
    assert len(waiting) >= 3  # tokens, tensor core, weights
    for role in waiting:
        # the wait ahead of a stage's first reuse stands inside that loop, and one before the epilogue serves short products
        assert re.search(r"g_pdl_wait(?:_only)?\(\)", role).start() < re.search(r"g_mbar_(?:wait|poll)", role).start(), role[:200]
    weights = waiting[2]
    assert weights.rindex("g_pdl_wait()") < weights.index("g_mbar_wait_warp(accum")
