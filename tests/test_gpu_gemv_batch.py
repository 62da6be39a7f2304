"""The matvec of 2..16 rows at the edges of its row groups, against 64-bit sums.

The activations are integers times a power of two with the largest quant in every 32-block, so that their 16-bit
quantization is exact and the result may differ from the 64-bit sum by the fp32 roundings of the fold only.
"""
import numpy as np
import pytest

import oracle
from litenn_b200 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FORMATS = {"q4_0": synth.Q4_0, "q8_0": synth.Q8_0, "q4_k": synth.Q4_K, "q6_k": synth.Q6_K}


def exact_activations(m, k, seed, one_sided):
    rng = np.random.default_rng(seed)
    q = rng.integers(0 if one_sided else -32639, 32640, size=(m, k // 32, 32))
    q[:, :, rng.integers(0, 32)] = 32639
    q[0, 0, :] = 32639 if one_sided else -32639  # every digit at its limit
    return (q * 2.0 ** -15 * 2.0 ** rng.integers(-3, 4, size=(m, k // 32, 1))).reshape(m, k).astype(np.float32)


def magnitudes(fmt, payload, n, k, w):
    """What the fold adds up, per weight: |w|, and for Q4_0 / Q4_K the offset that the kernel carries separately."""
    a = np.abs(w.astype(np.float64))
    if fmt == synth.Q4_K:
        blocks = payload.reshape(n, k // 256, 144)
        dmin = blocks[:, :, 2:4].copy().view(np.float16).astype(np.float64)[:, :, 0]
        s = blocks[:, :, 4:16].astype(np.int64)
        mins = np.concatenate([s[:, :, 4:8] & 63, (s[:, :, 8:12] >> 4) | ((s[:, :, 4:8] >> 6) << 4)], axis=2)
        a += 2.0 * np.repeat(np.abs(dmin[:, :, None] * mins), 32, axis=2).reshape(n, k)
    return a


@pytest.mark.parametrize("name", list(FORMATS))
@pytest.mark.parametrize("m", [2, 4, 5, 8, 9, 12, 13, 16])
@pytest.mark.parametrize("one_sided", [False, True])
def test_row_groups_against_64_bit(name, m, one_sided):
    fmt = FORMATS[name]
    unit = synth.BLOCK_ELEMS[fmt]
    for n, k in ((16, unit), (41, 256 * 3 + (unit if unit < 256 else 0)), (200, 256 * 11)):
        payload = synth.make_weight(fmt, n, k, seed=3, name="batch")
        w = oracle.dequant(fmt, payload, n, k)
        x = exact_activations(m, k, 7, one_sided)
        handle = capi.Weight.from_host(fmt, payload, n, k)
        xd = torch.from_numpy(x).cuda()
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        handle.gemv_f32(xd.data_ptr(), y.data_ptr(), m)
        torch.cuda.synchronize()
        handle.destroy()
        want = x.astype(np.float64) @ w.astype(np.float64).T
        # one rounding per sub-block's sum, scale product and addition, and the warps' sums; a term is added to at most
        # k / 16 + 8 others
        bound = (k / 16 + 16) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ magnitudes(fmt, payload, n, k, w).T)
        err = np.abs(y.cpu().numpy().astype(np.float64) - want)
        assert (err <= bound).all(), (name, m, n, k, float((err / bound).max()))
        # in the 2-norm the roundings average out: a few units of the last place
        assert np.linalg.norm(err) <= 1e-6 * np.linalg.norm(want) * (4.0 if fmt == synth.Q4_K else 2.0)
    assert capi.kernel_status(0) == 0


def test_a_row_keeps_its_infinities_to_itself():
    n, k, m = 32, 512, 7
    payload = synth.make_weight(synth.Q8_0, n, k, seed=3, name="batch")
    x = exact_activations(m, k, 7, False)
    bad = x.copy()
    bad[3, 40] = np.inf
    bad[4, 300] = np.nan
    handle = capi.Weight.from_host(synth.Q8_0, payload, n, k)
    out = []
    for v in (x, bad):
        xd = torch.from_numpy(v).cuda()
        y = torch.zeros((m, n), dtype=torch.float32, device="cuda")
        handle.gemv_f32(xd.data_ptr(), y.data_ptr(), m)
        torch.cuda.synchronize()
        out.append(y.cpu().numpy())
    handle.destroy()
    rows = [0, 1, 2, 5, 6]
    assert np.array_equal(out[0][rows], out[1][rows]) and not np.isfinite(out[1][3]).any()
