"""The matvec of one row over tiles per SM and chunks, for an fp32 vector (16-byte aligned and not) and a packed one.

Each size is the first row count whose tiles need `tiles` to an SM, with a ragged last tile, so that for an fp32 vector every
compiled number of tiles per CTA runs with most of its CTAs partly or wholly empty.  A packed vector takes small blocks for many
of these sizes; its one-wave forms are in test_gpu_gemv_wave_forms.py.
"""
import numpy as np
import pytest

import oracle
from litenn_b200 import capi, synth
from test_gpu_gemv_batch import FORMATS, exact_activations, magnitudes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# tiles per SM x chunks of 256 columns
SIZES = [(1, 1), (1, 4), (1, 5), (1, 33), (1, 113), (2, 8), (2, 17), (2, 33), (3, 4), (3, 5), (3, 9), (4, 3), (4, 17),
         (5, 2), (6, 8), (6, 9), (7, 8), (7, 9), (8, 8), (8, 9), (9, 2), (11, 1), (13, 2), (15, 1), (17, 1), (21, 1),
         (26, 1), (29, 1)]


@pytest.mark.parametrize("name", list(FORMATS))
@pytest.mark.parametrize("tiles,chunks", SIZES)
def test_tiles_per_sm_against_64_bit(name, tiles, chunks):
    fmt = FORMATS[name]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (sms * (tiles - 1) + 1) * 16 - 5
    k = chunks * 256 - (0 if synth.BLOCK_ELEMS[fmt] == 256 else 32)
    payload = synth.make_weight(fmt, n, k, seed=3, name="wave")
    w = oracle.dequant(fmt, payload, n, k)
    x = exact_activations(1, k, 7, False)
    handle = capi.Weight.from_host(fmt, payload, n, k)
    room = torch.empty(k + 4, dtype=torch.float32, device="cuda")
    y = torch.full((3, n + 8), float("nan"), dtype=torch.float32, device="cuda")
    for i, shift in enumerate((0, 1)):
        xd = room[shift:shift + k]
        xd.copy_(torch.from_numpy(x[0]))
        torch.cuda.synchronize()
        handle.gemv_f32(xd.data_ptr(), y[i].data_ptr(), 1)
        torch.cuda.synchronize()
    packed = torch.zeros(capi.packed_activation_bytes(k, 1), dtype=torch.uint8, device="cuda")
    capi.pack_activations(xd.data_ptr(), 1, k, packed.data_ptr())
    handle.gemv_packed(packed.data_ptr(), y[2].data_ptr(), 1)
    torch.cuda.synchronize()
    handle.destroy()
    assert torch.isnan(y[:, n:]).all()  # nothing beyond the last row
    x64, w64 = torch.from_numpy(x).cuda().double(), torch.from_numpy(w).cuda().double()
    want = (x64 @ w64.T)[0]
    mag = torch.from_numpy(magnitudes(fmt, payload, n, k, w)).cuda()
    # roundings of the fold as in the matvec of several rows
    bound = (k / 16 + 16) * 2.0 ** -24 * (x64.abs() @ mag.T)[0]
    err = (y[:, :n].double() - want).abs()
    assert bool((err <= bound).all()), (name, tiles, chunks, float((err / bound).max()))
    assert float(err.norm(dim=1).max() / want.norm()) <= 1e-6 * (4.0 if fmt == synth.Q4_K else 2.0)
    assert capi.kernel_status(0) == 0


def test_both_routes_take_what_is_not_finite_alike():
    """An infinity reaches every row; a NaN has no magnitude to scale by and counts as zero, in one launch as in two."""
    n, k = 100, 512
    payload = synth.make_weight(synth.Q8_0, n, k, seed=3, name="wave")
    handle = capi.Weight.from_host(synth.Q8_0, payload, n, k)
    room = torch.zeros(k + 4, dtype=torch.float32, device="cuda")
    y = torch.zeros(2, n, dtype=torch.float32, device="cuda")
    for bad in (float("inf"), float("nan"), 0.0):
        for i, shift in enumerate((0, 1)):
            room.copy_(torch.ones_like(room))
            room[shift + 40] = bad
            torch.cuda.synchronize()
            handle.gemv_f32(room[shift:].data_ptr(), y[i].data_ptr(), 1)
            torch.cuda.synchronize()
        if bad == float("inf"):
            assert not torch.isfinite(y).any()
        else:
            # two orders of the same sums of 16 blocks
            assert float((y[0] - y[1]).norm()) <= 16 * 2.0 ** -24 * float(y[1].norm())
    handle.destroy()
