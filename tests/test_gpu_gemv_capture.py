"""One-row products of both routes inside a stream capture, where nothing can be allocated."""
import pytest

from litenn_b200 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("warm", ["same weight", "other stream is captured"])
def test_a_call_before_the_capture_prepares_both_routes(warm):
    n, k = 512, 4096
    payload = synth.make_weight(synth.Q8_0, n, k, seed=5, name="capture")
    handle = capi.Weight.from_host(synth.Q8_0, payload, n, k)
    room = torch.zeros(k + 4, dtype=torch.float32, device="cuda")
    y = torch.zeros(3, n, dtype=torch.float32, device="cuda")
    x = room[1:k + 1]  # not on a 16-byte boundary: packed by a kernel of its own
    x.copy_(torch.from_numpy(synth.make_activation(1, k, seed=5, name="capture.x")[0]))
    packed = torch.zeros(capi.packed_activation_bytes(k, 1), dtype=torch.uint8, device="cuda")
    capi.pack_activations(x.data_ptr(), 1, k, packed.data_ptr())
    handle.gemv_packed(packed.data_ptr(), y[2].data_ptr(), 1)
    torch.cuda.synchronize()
    capi.check(capi.load().qmm_release_workspaces())
    stream, other, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    if warm == "same weight":
        handle.gemv_f32(room.data_ptr(), y[0].data_ptr(), 1, stream.cuda_stream)  # one launch
        torch.cuda.synchronize()
    else:  # the workspace of `stream` is made while another stream's capture is open
        with torch.cuda.graph(graph, stream=other):
            handle.gemv_f32(room.data_ptr(), y[1].data_ptr(), 1, other.cuda_stream)
            handle.gemv_f32(room.data_ptr(), y[0].data_ptr(), 1, stream.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y[0], y[1])
        graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        handle.gemv_f32(x.data_ptr(), y[1].data_ptr(), 1, stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    handle.destroy()
    assert torch.equal(y[1], y[2])
