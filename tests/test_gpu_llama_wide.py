"""Decoders wider than 4096 with few channels: both forms of their gate|up product, and its small blocks over long rows."""
import pytest

from litenn_b200 import capi, synth
from litenn_b200 import llama as ll
from test_gpu_llama import compare_with_oracle, stream  # noqa: F401  (fixture)
from test_gpu_parity import test_fused_swiglu_packed_output as check_gate_up
from test_gpu_parity import torch_cuda  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K])
@pytest.mark.parametrize("ffn", [512, 2304])  # fp32 from one row tile per block; packed, four warps per row tile
def test_decode_matches_oracle(stream, fmt, ffn):  # noqa: F811
    spec = ll.LlamaSpec(n_layers=2, d_model=4352, n_heads=4, n_kv_heads=2, head_dim=64, ffn=ffn, vocab=512, linear_fmt=fmt,
                        embd_fmt=synth.Q8_0, max_seq=64, max_prefill=32, unit_norms=False)
    compare_with_oracle(stream, spec, synth.make_token_ids(20, spec.vocab, seed=9, name="wide"), 8)


@pytest.mark.parametrize("fmt", [capi.Q4_0, capi.Q8_0, capi.Q4_K, capi.Q6_K])
# (64, 36864): no room for four warps per row tile of Q8_0; (64, 76032): for none of 1-byte and 6-bit tiles but one warp
@pytest.mark.parametrize("shape", [(2304, 4352), (64, 36864), (64, 76032)])
def test_gate_up_of_long_rows(torch_cuda, fmt, shape):  # noqa: F811
    check_gate_up(torch_cuda, fmt, shape)
