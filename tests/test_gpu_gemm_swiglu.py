"""The gate|up product of the prefill, bf16(silu(gate) * up) straight from the accumulators, in every form of the GEMM: its
epilogue pairs the 8 gates and 8 ups of a 16-row tile in registers, over a cluster's partial sums or along a row of the
accumulators, depending on the form.  Each form's fp32 product is checked against the oracle, and its fused result
against silu(gate) * up of that product."""
import ctypes

import numpy as np
import pytest

import native_build
import oracle
from litenn_b200 import capi, synth
from helpers import REL_TOL, max_rel_err

pytestmark = pytest.mark.gpu

GEMM_OUT_F32, GEMM_OUT_SWIGLU = 0, 2

# nb, tokens per CTA, K splits, keep_order; nb 0 is the shared-memory form
FORMS = [(1, 128, 1, 0), (1, 48, 2, 0), (1, 32, 4, 0), (1, 16, 8, 0), (1, 128, 8, 0), (2, 112, 1, 0), (2, 16, 1, 0),
         (0, 0, 1, 0), (0, 0, 1, 1)]


@pytest.fixture(scope="module")
def forms(qmm_lib):
    lib = native_build.load("gemm_forms", device_code=False, link_library=capi.LIB_PATH)
    lib.gemm_run_form.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int64] + [ctypes.c_int] * 5 + [ctypes.c_void_p]
    return lib


# 25 row tiles end inside a block of 8; K of 2080 is nine chunks, the last of 32 columns
@pytest.mark.parametrize("m,n,k", [(17, 16, 2080), (131, 400, 2080), (301, 400, 2304)])
@pytest.mark.parametrize("fmt", [capi.Q4_0, capi.Q8_0, capi.Q4_K, capi.Q6_K])
@pytest.mark.parametrize("nb,tokens,splits,keep", FORMS)
def test_fused_result_is_silu_gate_times_up(forms, nb, tokens, splits, keep, fmt, m, n, k):
    import torch
    unit = synth.BLOCK_ELEMS[fmt]
    k = (k + unit - 1) // unit * unit
    payload = synth.make_weight(fmt, n, k, seed=9, name=f"glu-{fmt}-{n}-{k}")
    w = capi.Weight.from_host(fmt, payload, n, k)
    x = torch.from_numpy(synth.make_activation(m, k, seed=9, name=f"glu-x-{m}")).cuda().to(torch.bfloat16).contiguous()
    y = torch.full((m * n + n,), 7.0, device="cuda")
    act = torch.full((m * n // 2 + n,), 7.0, device="cuda", dtype=torch.bfloat16)
    for out, buf in ((GEMM_OUT_F32, y), (GEMM_OUT_SWIGLU, act)):
        assert forms.gemm_run_form(w.handle, x.data_ptr(), buf.data_ptr(), m, out, nb, tokens, splits, keep, None) == 0
    torch.cuda.synchronize()
    assert capi.kernel_status(0) == 0
    assert bool((y[m * n:] == 7.0).all()) and bool((act[m * n // 2:] == 7.0).all())
    product = y[:m * n].view(m, n).cpu().numpy()
    ref = oracle.matmul_nk_f64(x.float().cpu().numpy(), oracle.fp32_to_bf16_round(oracle.dequant(fmt, payload, n, k)))
    assert max_rel_err(product, ref) <= REL_TOL
    pairs = product.astype(np.float64).reshape(m, n // 16, 2, 8)  # a row tile: 8 gates, then their 8 ups
    gate, up = pairs[:, :, 0], pairs[:, :, 1]
    want = (gate / (1.0 + np.exp(-gate)) * up).reshape(m, n // 2)
    got = act[:m * n // 2].view(m, n // 2).float().cpu().numpy()
    # one bf16 rounding (8 bits: 2^-8 relative at most) behind fp32 arithmetic, whose exp(-gate) overflows beyond 88.7:
    # what is lost there is 89 * exp(-88.7) = 3e-37 of up
    bound = 2.0 ** -8 * 1.001 * np.abs(want) + 1e-36 * (1.0 + np.abs(up).reshape(m, n // 2))
    assert (np.abs(got - want) <= bound).all()
