"""Prefill attention inside a model, with a cache that already holds an earlier piece of the prompt, for both head sizes and
grouped heads, against the numpy oracle.  Narrow models take the fp32 row kernel up to 256 rows; the wide ones here take
the tensor-core kernel from 33 rows on, at the edges of its tiles (16 rows per warp, 64 rows per CTA, 64 keys per tile).
test_gpu_prefill_attention_tiles.py looks at the kernels by themselves."""
import numpy as np
import pytest

from litenn_b200 import capi, synth
from litenn_b200 import llama as ll

pytestmark = pytest.mark.gpu

# The bar of the other prefill tests: both sides round activations and weights to bf16 at the same points, and a last-bit
# difference of a sum flips some of those roundings (2^-8 relative each) between the layers.
TOL = 1e-2


def check(spec, pieces):
    import torch
    from oracle.llama_ref import LlamaOracle
    stream = torch.cuda.Stream()
    model = ll.LlamaModel(spec, stream=stream.cuda_stream, seed=3)
    ref = LlamaOracle(spec, seed=3)
    tokens = synth.make_token_ids(sum(pieces), spec.vocab, seed=3, name="pieces")
    at = 0
    for n in pieces:
        model.prefill(tokens[at:at + n])
        ref.prefill(tokens[at:at + n])
        at += n
        err = np.abs(model.last_logits() - ref.last_logits).max() / np.abs(ref.last_logits).max()
        assert err <= TOL, (at, err)
    assert capi.kernel_status(0) == 0
    model.close()


@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 4, 2), (128, 4, 1), (128, 2, 2)])
@pytest.mark.parametrize("pieces", [[1], [15], [16, 1], [17, 46], [63], [64], [65], [1, 64, 63], [64, 64, 2], [150, 107]],
                         ids=lambda p: "+".join(map(str, p)))
def test_prompt_pieces_match_oracle(qmm_lib, head_dim, heads, kv_heads, pieces):
    check(ll.LlamaSpec(n_layers=2, d_model=256, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, ffn=512, vocab=512,
                       linear_fmt=synth.Q8_0, embd_fmt=synth.Q6_K, max_seq=sum(pieces), max_prefill=max(pieces),
                       unit_norms=False), pieces)


@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 36, 9), (128, 18, 18)])
@pytest.mark.parametrize("pieces", [[33], [63], [65], [64, 65], [100, 157]], ids=lambda p: "+".join(map(str, p)))
def test_prompt_pieces_of_a_wide_model_match_oracle(qmm_lib, head_dim, heads, kv_heads, pieces):
    check(ll.LlamaSpec(n_layers=1, d_model=2304, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, ffn=512, vocab=512,
                       linear_fmt=synth.Q8_0, embd_fmt=synth.Q6_K, max_seq=sum(pieces), max_prefill=max(pieces),
                       unit_norms=False), pieces)
