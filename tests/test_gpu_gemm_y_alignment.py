"""Results of the prefill GEMM at every element address a caller may hand over (a row or a column of a larger buffer): the
shared-memory form stores sixteen bytes at a time where the address allows it and single elements elsewhere, with the
same bits; the other forms store single elements."""
import numpy as np
import pytest

from litenn_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out_bf16", [False, True], ids=["f32", "bf16"])
@pytest.mark.parametrize("m,n,k", [(700, 8192, 256), (300, 14344, 288), (33, 128, 1024), (131, 12296, 288)])
def test_any_result_address_gives_the_same_bits(qmm_lib, m, n, k, out_bf16):
    import torch
    payload = synth.make_weight(capi.Q8_0, n, k, seed=6, name="ypos")
    w = capi.Weight.from_host(capi.Q8_0, payload, n, k)
    x = torch.from_numpy(synth.make_activation(m, k, seed=6, name="ypos.x")).cuda().to(torch.bfloat16).contiguous()
    dtype, code = (torch.bfloat16, capi.OUT_BF16) if out_bf16 else (torch.float32, capi.OUT_F32)
    per16 = 8 if out_bf16 else 4
    want = None
    for shift in range(per16):
        room = torch.full((m * n + 2 * per16,), 7.0, device="cuda", dtype=dtype)
        w.gemm_bf16(x.data_ptr(), room[shift:].data_ptr(), m, code)
        torch.cuda.synchronize()
        got = room[shift:shift + m * n].float().cpu().numpy()
        assert bool((room[:shift] == 7.0).all()) and bool((room[shift + m * n:] == 7.0).all()), shift
        want = got if want is None else want
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), shift
    assert capi.kernel_status(0) == 0
