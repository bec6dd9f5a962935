"""Cast to e4m3 on the GPU, with and without saturation: every 16-bit value, and lengths around the vector width, byte for byte as the
tensor library converts (what saturates beforehand); every run is one launch of the kernel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _session(dtype, saturate):
    import onnxruntime_b200 as ort
    from onnxruntime_b200 import onnx_lite as ol
    P = ol.TensorProto
    graph = ol.make_graph([ol.make_node("Cast", ["x"], ["y"], to=P.FLOAT8E4M3FN, saturate=saturate)], "cast", [ol.make_tensor_value_info("x", dtype, ["n"])],
                          [ol.make_tensor_value_info("y", P.FLOAT8E4M3FN, ["n"])], [])
    return ort.InferenceSession(ol.make_model(graph, opset=19).serialize(), providers=[("CUDAExecutionProvider", {})], enable_fallback=False)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("saturate", [1, 0])
def test_every_value(bf16, saturate):
    from onnxruntime_b200 import onnx_lite as ol
    sess = _session(ol.TensorProto.BFLOAT16 if bf16 else ol.TensorProto.FLOAT16, saturate)
    bits = torch.arange(65536, dtype=torch.int32).to(torch.int16).cuda()
    x = bits.view(torch.bfloat16 if bf16 else torch.float16)
    want = (x.clamp(-448, 448) if saturate else x).to(torch.float8_e4m3fn).view(torch.uint8)
    for n in (65536, 1, 7, 8, 9, 2047, 2048, 2049):
        for start in (0, 65536 - n):
            part = x[start:start + n].clone()
            out = torch.zeros(n, dtype=torch.float8_e4m3fn, device="cuda")
            binding = sess.io_binding()
            binding.bind_torch_input("x", part)
            binding.bind_torch_output("y", out)
            before = sess.kernel_launch_count()
            sess.run_with_iobinding(binding, None)
            assert sess.kernel_launch_count() == before + 1
            torch.cuda.synchronize()
            got = out.view(torch.uint8)
            assert torch.equal(got, want[start:start + n]), np.flatnonzero((got != want[start:start + n]).cpu().numpy())[:8]
