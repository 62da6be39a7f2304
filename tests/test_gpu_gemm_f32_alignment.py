"""fp32 activations of the prefill GEMM at every alignment a caller may have: rows that start on a 16-byte boundary take
the vector conversion, others the scalar one, and both round alike."""
import numpy as np
import pytest

from litenn_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(17, 48, 32), (77, 130, 1312), (300, 64, 256)])
def test_any_alignment_gives_the_same_bits(qmm_lib, m, n, k):
    import torch
    payload = synth.make_weight(capi.Q8_0, n, k, seed=2, name="align")
    w = capi.Weight.from_host(capi.Q8_0, payload, n, k)
    x = torch.from_numpy(synth.make_activation(m, k, seed=2, name="align.x")).cuda()
    xb = x.to(torch.bfloat16).contiguous()
    want = torch.empty((m, n), device="cuda")
    w.gemm_bf16(xb.data_ptr(), want.data_ptr(), m)
    room = torch.empty(m * k + 8, device="cuda")
    for shift in range(4):
        room[shift:shift + m * k] = x.view(-1)
        got = torch.empty((m, n), device="cuda")
        w.gemm_f32(room[shift:].data_ptr(), got.data_ptr(), m)
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy().view(np.uint32), want.cpu().numpy().view(np.uint32)), shift
    assert capi.kernel_status(0) == 0
