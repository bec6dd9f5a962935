"""GEMM on CTA pairs: the order of its tiles (runs of token tiles, uneven experts), the two epilogue groups and the gated
epilogue, at edges of token tiles, weight tiles and runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _limit(z, dtype, Kd, scale=1.0):
    # half a unit in the last place of the result, and fp32 sums of Kd products of magnitude 0.05
    return z.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01 + 2.0 ** -20 * Kd ** 0.5 * scale


@pytest.mark.parametrize("M,N,Kd", [(512, 264, 512), (700, 1000, 200), (2561, 260, 64), (2816, 1027, 1160), (5377, 256, 72)])
@pytest.mark.parametrize("act", ["none", "relu", "swiglu", "geglu"])
def test_pair_gemm(M, N, Kd, act):
    from onnxruntime_b200.ops import _kernels as K
    dtype = torch.float16 if M % 2 else torch.bfloat16
    gated = act in ("swiglu", "geglu")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w = rand(M, Kd).to(dtype), (rand(N * (2 if gated else 1), Kd) * 0.05).to(dtype)
    bias, residual = (None, None) if gated else (rand(N).to(dtype), rand(M, N).to(dtype))
    y = K.gemm(x, w, bias=bias, residual=residual, act=act, force_tile_rows=512)
    z = x.double() @ w.double().t()
    if gated:
        a, b = z[:, :N], z[:, N:]
        z = (torch.nn.functional.silu(a) if act == "swiglu" else torch.nn.functional.gelu(a, approximate="tanh")) * b
        # gate and up are in error by up to 2^-20 sqrt(Kd) each, times the other factor (below 10 here)
        assert ((y.double() - z).abs() <= _limit(z, dtype, Kd, 10)).all()
        return
    z = z + bias.double()
    z = z.relu() if act == "relu" else z
    total = z + residual.double()
    # the staged value is rounded to 16 bits before the activation and the residual, and the sum is rounded again
    assert ((y.double() - total).abs() <= _limit(total, dtype, Kd) + _limit(z, dtype, Kd)).all()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_pair_gemm_gated_keeps_special_values(value):
    from onnxruntime_b200.ops import _kernels as K
    x, w = torch.zeros(512, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(512, 64, device="cuda", dtype=torch.bfloat16)
    x[:, 0], x[7, 0], w[:, 0] = 1.0, value, 1.0
    y = K.gemm(x, w, act="swiglu", force_tile_rows=512)
    a = (x.float() @ w[:256].float().t())
    z = torch.nn.functional.silu(a) * a
    assert torch.equal(torch.isnan(y), torch.isnan(z))
    assert torch.equal(torch.isinf(y), torch.isinf(z))


@pytest.mark.parametrize("counts", [(2700, 299, 1, 0), (0, 5, 2995, 0), (750, 750, 750, 750)])
def test_grouped_pair_gemm_runs(counts):
    import onnxruntime_b200 as ort
    from onnxruntime_b200 import onnx_lite as ol
    E, H, F, T = 4, 256, 264, sum(counts)
    g = torch.Generator(device="cuda").manual_seed(T + counts[0])
    bf16 = torch.bfloat16
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w1, w2, w3 = rand(T, H).to(bf16), (rand(E, F, H) * 0.05).to(bf16), (rand(E, H, F) * 0.05).to(bf16), (rand(E, F, H) * 0.05).to(bf16)
    chosen = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=torch.Generator().manual_seed(1))].cuda()
    router = torch.zeros(T, E, device="cuda", dtype=bf16)
    router[torch.arange(T, device="cuda"), chosen] = 8.0
    P = ol.TensorProto
    node = ol.make_node("MoE", ["x", "router", "fc1", "", "fc2", "", "fc3"], ["y"], domain="com.microsoft", k=1, activation_type="silu", normalize_routing_weights=1)
    info = lambda n, c: ol.make_tensor_value_info(n, P.BFLOAT16, ["tokens", c])  # noqa: E731
    weights = {"fc1": w1, "fc2": w2, "fc3": w3}
    graph = ol.make_graph([node], "moe", [info("x", H), info("router", E)], [info("y", H)],
                          [ol.make_external_tensor(n, P.BFLOAT16, list(w.shape)) for n, w in weights.items()])
    so = ort.SessionOptions()
    so.add_external_initializers(list(weights), list(weights.values()))
    sess = ort.InferenceSession(ol.make_model(graph).serialize(), so, providers=[("CUDAExecutionProvider", {})], enable_fallback=False)
    out = torch.full_like(x, float("nan"))
    binding = sess.io_binding()
    binding.bind_torch_input("x", x)
    binding.bind_torch_input("router", router)
    binding.bind_torch_output("y", out)
    sess.run_with_iobinding(binding, None)
    torch.cuda.synchronize()
    sess.check_device_status()
    z = torch.empty(T, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        rows = (chosen == e).nonzero(as_tuple=True)[0]
        d = x[rows].double()
        z[rows] = (torch.nn.functional.silu(d @ w1[e].double().t()) * (d @ w3[e].double().t())) @ w2[e].double().t()
    # the hidden values are rounded to 8 bits (2^-9 relative each, over a sum of F of them), the result twice
    rms = float(z.square().mean().sqrt())
    assert (out.double() - z).abs().max() <= 2.0 ** -8 * (2 * float(z.abs().max()) + 6 * rms)
