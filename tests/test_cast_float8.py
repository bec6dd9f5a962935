"""Cast, CastLike and QuantizeLinear to the 8-bit float types: what lies beyond the largest number with and without ``saturate``
(1 unless given), from every float type and from integers."""
import numpy as np
import pytest
import torch

import onnxruntime_b200 as ort
from onnxruntime_b200 import onnx_lite as ol

P = ol.TensorProto
TYPES = {P.FLOAT8E4M3FN: (torch.float8_e4m3fn, 448.0), P.FLOAT8E4M3FNUZ: (torch.float8_e4m3fnuz, 240.0),
         P.FLOAT8E5M2: (torch.float8_e5m2, 57344.0), P.FLOAT8E5M2FNUZ: (torch.float8_e5m2fnuz, 57344.0)}
PROVIDERS = [["CPUExecutionProvider"], pytest.param([("CUDAExecutionProvider", {})], marks=pytest.mark.gpu)]
VALUES = [0.0, 1.0, -1.0625, 239.0, 240.0, 256.0, 447.0, 448.0, 460.0, -464.0, 465.0, -500.0, 50000.0, 57344.0, 61000.0, 65504.0, float("inf"),
          float("-inf"), float("nan")]


def _run(providers, op, source, to, attrs, values):
    inputs, extra = [ol.make_tensor_value_info("x", source, ["n"])], []
    if op == "CastLike":
        inputs.append(ol.make_tensor_value_info("like", to, [1]))
        extra = ["like"]
    elif op == "QuantizeLinear":
        inputs.append(ol.make_tensor_value_info("scale", P.FLOAT, []))
        extra, attrs = ["scale"], dict(attrs, output_dtype=to)
    else:
        attrs = dict(attrs, to=to)
    nodes = [ol.make_node(op, ["x"] + extra, ["y8"], **attrs), ol.make_node("Cast", ["y8"], ["y"], to=P.FLOAT)]
    graph = ol.make_graph(nodes, "cast", inputs, [ol.make_tensor_value_info("y", P.FLOAT, ["n"])], [])
    sess = ort.InferenceSession(ol.make_model(graph, opset=21).serialize(), providers=providers)
    binding = sess.io_binding()
    dev = "cpu" if providers == ["CPUExecutionProvider"] else "cuda"
    feeds = {"x": values.to(dev)}
    if op == "CastLike":
        feeds["like"] = torch.zeros(1).to(TYPES[to][0]).to(dev)
    elif op == "QuantizeLinear":
        feeds["scale"] = torch.tensor(1.0, device=dev)
    out = torch.zeros(values.numel(), device=dev)
    for name, t in feeds.items():
        binding.bind_torch_input(name, t)
    binding.bind_torch_output("y", out)
    sess.run_with_iobinding(binding, None)
    if dev == "cuda":
        torch.cuda.synchronize()
    return out.cpu()


@pytest.mark.parametrize("providers", PROVIDERS)
@pytest.mark.parametrize("op", ["Cast", "CastLike", "QuantizeLinear"])
@pytest.mark.parametrize("to", list(TYPES))
@pytest.mark.parametrize("saturate", [None, 1, 0])
@pytest.mark.parametrize("source,dtype", [(P.FLOAT, torch.float32), (P.FLOAT16, torch.float16), (P.BFLOAT16, torch.bfloat16)])
def test_beyond_the_largest_number(providers, op, to, saturate, source, dtype):
    kind, largest = TYPES[to]
    x = torch.tensor(VALUES).to(dtype)
    got = _run(providers, op, source, to, {} if saturate is None else {"saturate": saturate}, x)
    want = x.float()
    if saturate != 0:
        want = torch.where(want.abs() > largest, torch.sign(want) * largest, want)   # NaN compares false and stays
    want = want.to(kind).float()
    if saturate == 0:
        assert not torch.isfinite(want[-3:]).any()
    np.testing.assert_array_equal(got.numpy(), want.numpy())


@pytest.mark.parametrize("providers", PROVIDERS)
def test_integers_saturate(providers):
    x = torch.tensor([0, 1, -3, 448, 449, 100000, -100000], dtype=torch.int32)
    got = _run(providers, "Cast", P.INT32, P.FLOAT8E4M3FN, {}, x)
    np.testing.assert_array_equal(got.numpy(), [0, 1, -3, 448, 448, 448, -448])
