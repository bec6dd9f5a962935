"""Epilogue of the decode-shaped GEMM: which CTA of a cluster finishes (and normalises) which token column, four weight rows
per lane with and without aligned 8-byte stores, at the edges of the column and row tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 17, 33, 40, 64])
@pytest.mark.parametrize("N,Kd", [(128, 512), (1003, 768), (1026, 2056), (260, 4096)])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("gated,rms", [(False, 0.0), (False, 1e-5), (True, 1e-5)])
def test_decode_gemm_epilogue(M, N, Kd, splits, gated, rms):
    from onnxruntime_b200.ops import _kernels as K
    dtype = torch.float16 if N % 2 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N + splits)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w = rand(M, Kd).to(dtype), (rand(N * (2 if gated else 1), Kd) * 0.05).to(dtype)
    bias = None if gated else rand(N).to(dtype)
    residual = rand(M, N + 4).to(dtype)[:, 1:N + 1] if N % 4 == 0 else rand(M, N).to(dtype)   # rows that are not 8-byte aligned, and that are
    y = K.gemm(x, w, bias=bias, residual=residual, act="swiglu" if gated else "none", rms_eps=rms, force_splits=splits)
    d = x.double()
    scale = torch.rsqrt(d.square().mean(-1, keepdim=True) + rms) if rms else 1.0
    z = d @ w.double().t() * scale
    if gated:
        a, b = z[:, :N], z[:, N:]
        z = torch.nn.functional.silu(a) * b
    else:
        z = z + bias.double()
    z = z + residual.double()
    # half a unit in the last place of the result (8 or 11 significant bits: at most 2^-8 or 2^-11 of the value), and fp32 sums of Kd products of magnitude 0.05 (times the other factor of the gated form)
    limit = z.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01 + 2.0 ** -20 * Kd ** 0.5 * (10 if gated else 1)
    assert ((y.double() - z).abs() <= limit).all()
