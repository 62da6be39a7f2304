"""One row times a weight with the result over the activations, wholly or in part: the same bits as from a buffer of its own."""
import pytest

from litenn_b200 import capi, synth
from test_gpu_gemv_batch import FORMATS

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", list(FORMATS))
@pytest.mark.parametrize("shift", [0, 1])  # x on a 16-byte boundary and beside one
@pytest.mark.parametrize("n,k,to_y", [(4096, 4096, 0), (4096, 4096, 2050), (4096, 4096, -4095), (2304, 1024, -700),
                                      (1024, 4096, 3072)])
def test_result_over_the_activations(name, shift, n, k, to_y):
    payload = synth.make_weight(FORMATS[name], n, k, seed=5, name="in place")
    handle = capi.Weight.from_host(FORMATS[name], payload, n, k)
    room = torch.zeros(2 * n + k + 8, dtype=torch.float32, device="cuda")
    x = room[n + shift:n + shift + k]
    x.copy_(torch.from_numpy(synth.make_activation(1, k, seed=5, name="in place.x")[0]))
    torch.cuda.synchronize()
    assert (x.data_ptr() % 16 == 0) == (shift == 0)
    want = torch.empty(n, dtype=torch.float32, device="cuda")
    packed = torch.zeros(capi.packed_activation_bytes(k, 1), dtype=torch.uint8, device="cuda")
    capi.pack_activations(x.data_ptr(), 1, k, packed.data_ptr())
    handle.gemv_packed(packed.data_ptr(), want.data_ptr(), 1)
    torch.cuda.synchronize()
    y = room[n + shift + to_y:n + shift + to_y + n]
    handle.gemv_f32(x.data_ptr(), y.data_ptr(), 1)
    torch.cuda.synchronize()
    handle.destroy()
    assert torch.equal(y, want)
