"""The prefill GEMM's CTA shapes at their edges: K split over a cluster of 2, 4 or 8, one or two blocks of 128 weight rows
per CTA, and the shared-memory form; row counts around the 16-token granule and the 128- and 256-token tiles, weight
rows that end inside a 16-row tile, K that ends inside a 256-wide chunk.  The shapes are sized so that the dispatch
reaches the named form on a 148-SM part (test_gemm_plan.py holds it to that); on another part they still have to be
right."""
import numpy as np
import pytest

import oracle
from litenn_b200 import capi, synth
from helpers import REL_TOL, max_rel_err

pytestmark = pytest.mark.gpu

CASES = [
    # form, m, n, k (k is rounded to whole super-blocks for the K-quants)
    ("one CTA per tile", 17, 3, 32),
    ("split", 16, 40, 1056), ("split", 33, 129, 1024), ("split", 128, 1000, 2080), ("split", 129, 250, 2048),
    ("split, several token tiles", 250, 520, 1312),
    ("two blocks", 131, 12291, 288), ("two blocks", 145, 14344, 256),
    ("shared memory", 257, 14347, 288), ("shared memory", 700, 8193, 256), ("shared memory", 2050, 2305, 544),
]


@pytest.mark.parametrize("out_bf16", [False, True], ids=["f32", "bf16"])
@pytest.mark.parametrize("fmt", [capi.Q4_0, capi.Q8_0, capi.Q4_K, capi.Q6_K])
@pytest.mark.parametrize("form,m,n,k", CASES)
def test_every_cta_shape_matches_oracle(qmm_lib, form, m, n, k, fmt, out_bf16):
    import torch
    unit = synth.BLOCK_ELEMS[fmt]
    k = (k + unit - 1) // unit * unit
    payload = synth.make_weight(fmt, n, k, seed=21, name=f"forms-{fmt}-{n}-{k}")
    x = synth.make_activation(m, k, seed=21, name=f"forms-x-{m}")
    w = capi.Weight.from_host(fmt, payload, n, k)
    xb = torch.from_numpy(x).cuda().to(torch.bfloat16).contiguous()
    # one row and one column more than the product: nothing may be written outside of it
    y = torch.full((m * n + n + 1,), 7.0, device="cuda", dtype=torch.bfloat16 if out_bf16 else torch.float32)
    w.gemm_bf16(xb.data_ptr(), y.data_ptr(), m, capi.OUT_BF16 if out_bf16 else capi.OUT_F32)
    torch.cuda.synchronize()
    assert capi.kernel_status(0) == 0
    assert bool((y[m * n:] == 7.0).all())
    got = y[:m * n].view(m, n).float().cpu().numpy()
    rng = np.random.default_rng(5)
    rows = np.unique(np.concatenate([[0, n - 1], rng.choice(n, size=min(n, 200), replace=False)]))
    rb = k // unit * synth.BLOCK_BYTES[fmt]
    sub = np.concatenate([payload[r * rb:(r + 1) * rb] for r in rows])
    ref = oracle.matmul_nk_f64(xb.float().cpu().numpy(), oracle.fp32_to_bf16_round(oracle.dequant(fmt, sub, len(rows), k)))
    # fp32 accumulation in the tensor core against 64 bits; bf16 results are rounded once more (2^-8 relative)
    assert max_rel_err(got[:, rows], ref) <= (5e-3 if out_bf16 else REL_TOL)
