"""Every compiled one-wave form of the one-row matvec, plain and fused, against 64-bit sums.

The shapes come from the rules themselves: the smallest that takes a form, and the smallest whose warps also refill their
slots.  The weight repeats 257 rows, so that no tile equals its neighbours.
"""
import ctypes

import numpy as np
import pytest

import native_build
from litenn_b200 import capi, synth
from test_gpu_gemv_batch import FORMATS, exact_activations

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STORE, RESIDUAL, GATE_UP = 0, 1, 3
PERIOD = 257


@pytest.fixture(scope="module")
def lib(qmm_lib):
    return native_build.load("gemv_route", device_code=False, link_library=capi.LIB_PATH)


def shapes_of(lib, fmt, epi, xf32):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    out = (ctypes.c_int * (6 * 256))()
    count = lib.gemv_wave_shapes(fmt, epi, xf32, sms, out, 256)
    assert 0 < count < 256
    return sorted({tuple(out[6 * i:6 * i + 6]) for i in range(count)})


def device_weight(fmt, n, k):
    base = torch.from_numpy(synth.make_weight(fmt, PERIOD, k, seed=11, name="forms")).cuda().reshape(PERIOD, -1)
    payload = base[torch.arange(n, device="cuda") % PERIOD].contiguous()
    handle = capi.Weight.from_device(fmt, payload.data_ptr(), payload.numel(), n, k)
    rows = capi.Weight.from_device(fmt, base.data_ptr(), base.numel(), PERIOD, k)
    w = torch.empty(PERIOD, k, dtype=torch.float32, device="cuda")
    rows.dequantize(w.data_ptr())
    torch.cuda.synchronize()
    rows.destroy()
    return handle, w.double()


def pack(x):
    out = torch.zeros(capi.packed_activation_bytes(x.numel(), 1), dtype=torch.uint8, device="cuda")
    capi.pack_activations(x.data_ptr(), 1, x.numel(), out.data_ptr())
    return out


def close(got, want, fmt):
    # fp32 roundings of the fold, as in the matvecs' own tests; Q4_K adds its offsets separately
    return float((got.double() - want).norm() / want.norm()) <= 1e-6 * (4.0 if fmt == synth.Q4_K else 2.0)


def packed_as(packed, values):
    """The record holds the values within half a step of their 32-wide block's 16-bit quantization."""
    back = torch.empty(values.numel(), dtype=torch.float32, device="cuda")
    capi.unpack_activations(packed.data_ptr(), values.numel(), back.data_ptr())
    v = values.reshape(-1, 32)
    step = v.abs().amax(dim=1, keepdim=True) / 32639.0
    return bool(((back.reshape(-1, 32) - v).abs() <= 0.51 * step + 1e-30).all())


@pytest.mark.parametrize("epi,xf32", [(STORE, 1), (STORE, 0), (RESIDUAL, 0), (GATE_UP, 0)],
                         ids=["fp32 vector", "packed vector", "residual", "gate|up"])
@pytest.mark.parametrize("name", list(FORMATS))
def test_form(lib, name, epi, xf32):
    fmt = FORMATS[name]
    for tiles, warps, depth, rt, kc, chained in shapes_of(lib, fmt, epi, xf32):
        what = (name, tiles, warps, depth, rt, kc)
        n = rt * 16 - (5 if epi == STORE else 0)
        k = kc * 256 - (0 if synth.BLOCK_ELEMS[fmt] == 256 else 32)
        handle, w = device_weight(fmt, n, k)
        x = torch.from_numpy(exact_activations(1, k, 7, False)[0]).cuda()
        order = torch.arange(n, device="cuda") % PERIOD
        product = (w @ x.double())[order]
        packed = pack(x)
        y = torch.full((n + 64,), float("nan"), dtype=torch.float32, device="cuda")
        ss = (x.double().reshape(-1, 32) ** 2).sum(dim=1)
        rms = float(torch.sqrt(ss.sum() / k + 1e-6))
        if epi == STORE:
            if xf32:
                handle.gemv_f32(x.data_ptr(), y.data_ptr(), 1)
            elif chained:
                handle.gemv_packed_rms(packed.data_ptr(), ss.data_ptr(), k // 32, k, 1e-6, y.data_ptr())
                product = product / rms
            else:
                handle.gemv_packed(packed.data_ptr(), y.data_ptr(), 1)
            torch.cuda.synchronize()
            assert close(y[:n], product, fmt), what
            assert torch.isnan(y[n:]).all(), what
        elif epi == RESIDUAL:
            h = torch.arange(n, device="cuda", dtype=torch.float32) / n * float(product.abs().max())
            want = h.double() + product
            norm = 1.0 + torch.arange(n, device="cuda", dtype=torch.float32) / n
            record, squares = pack(torch.zeros_like(h)), torch.full((n // 32,), -1.0, dtype=torch.float64, device="cuda")
            handle.gemv_packed_residual(packed.data_ptr(), h.data_ptr(), norm.data_ptr(), record.data_ptr(), squares.data_ptr())
            torch.cuda.synchronize()
            assert close(h, want, fmt), what
            assert packed_as(record, h * norm), what
            assert torch.allclose(squares, (h.double().reshape(-1, 32) ** 2).sum(dim=1), rtol=1e-12), what
        else:
            gate, up = (product / rms).reshape(-1, 2, 8).unbind(dim=1)  # rows alternate eight of gate and eight of up
            want = (gate * torch.sigmoid(gate) * up).reshape(-1)
            record = pack(torch.zeros(n // 2, dtype=torch.float32, device="cuda"))
            handle.gemv_packed_swiglu_pack(packed.data_ptr(), ss.data_ptr(), k // 32, k, 1e-6, record.data_ptr(), y.data_ptr())
            torch.cuda.synchronize()
            # relative errors of gate and up add, and silu grows by at most 1.1 per unit of its argument
            scale = float((gate.abs().max() + 2.0) * 4e-6 * (2.0 if fmt == synth.Q4_K else 1.0))
            assert float((y[:n // 2].double() - want).norm() / want.norm()) <= scale, what
            assert torch.isnan(y[n // 2:]).all(), what
            assert packed_as(record, y[:n // 2].clone()), what
        handle.destroy()
    assert capi.kernel_status(0) == 0
