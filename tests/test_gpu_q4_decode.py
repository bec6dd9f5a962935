"""Decode GEMM on packed 4-bit weights, up to 16 tokens on warp-level products and above on tcgen05: edges of token tiles, row tiles and splits of K (odd numbers of
64-wide blocks among them), bias, residual and output rows with and without 8-byte alignment, against 64-bit products of the
dequantised weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("N,Kd", [(128, 64), (1003, 192), (260, 1088), (1026, 2112), (384, 4096)])
@pytest.mark.parametrize("splits", [0, 1, 2, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_q4_decode(M, N, Kd, splits, dtype):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N)
    B = torch.randint(0, 256, (N, Kd // 32, 16), generator=g, device="cuda", dtype=torch.uint8)
    scales = (torch.rand(N, Kd // 32, generator=g, device="cuda") * 0.02 + 0.001).to(dtype)
    zp = torch.randint(0, 16, (N, Kd // 32), generator=g, device="cuda", dtype=torch.uint8)
    blobs = K.nbits_build_blobs(B, scales, zp, N, Kd, 32)
    q = torch.stack([B & 15, B >> 4], -1).reshape(N, Kd // 32, 32).float() - zp.float().unsqueeze(-1)
    w = (q * scales.float().unsqueeze(-1)).to(dtype).reshape(N, Kd).double()     # the product rounded to 16 bits, as the kernel does
    x = torch.randn(M, Kd, generator=g, device="cuda").to(dtype)
    bias = torch.randn(N, generator=g, device="cuda").to(dtype)
    wide = torch.randn(M, N + 4, generator=g, device="cuda").to(dtype)
    residual = wide[:, 1:N + 1] if N % 4 == 0 else wide[:, :N].contiguous()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    y = K.gemm(x, blobs, bias=bias, residual=residual, n=N, q4=True, force_splits=splits, status=status)
    z = x.double() @ w.t() + bias.double() + residual.double()
    # half a unit in the last place of the result, and fp32 sums of Kd products of magnitude up to 0.3
    limit = z.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01 + 2.0 ** -20 * Kd ** 0.5 * 6
    assert status.item() == 0
    assert ((y.double() - z).abs() <= limit).all()
