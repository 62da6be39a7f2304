"""What the prefill GEMM refuses, and that the message names the offending value."""
import pytest

from litenn_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,out_dtype,text", [(0, capi.OUT_F32, "invalid row count 0"), (4, 2, "unknown output type 2"),
                                              (4, -1, "unknown output type -1"), (0, 7, "invalid row count 0")])
def test_bad_arguments_are_named(qmm_lib, m, out_dtype, text):
    import torch
    w = capi.Weight.from_host(capi.Q8_0, synth.make_weight(capi.Q8_0, 16, 32, seed=1, name="refuse"), 16, 32)
    x = torch.zeros(4, 32, device="cuda", dtype=torch.bfloat16)
    y = torch.full((4, 16), 7.0, device="cuda")
    with pytest.raises(capi.QmmError) as e:
        w.gemm_bf16(x.data_ptr(), y.data_ptr(), m, out_dtype)
    torch.cuda.synchronize()
    assert e.value.code == capi.E_INVALID and text in str(e.value)
    assert bool((y == 7.0).all())
