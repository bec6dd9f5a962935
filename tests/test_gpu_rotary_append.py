"""Rotary embedding and cache append by 16-byte vectors against the pair-by-pair path (the same call on views that are not
16-byte aligned) and a 32-bit restatement: head sizes on and off the vector path, few and many tokens, no rotation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _shifted(t):
    """The same values two bytes off a 16-byte boundary."""
    base = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    view = base[1:1 + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("H", [16, 48, 64, 96, 128, 256, 72])
@pytest.mark.parametrize("B,S,past", [(1, 1, 5), (3, 7, 0), (2, 200, 30)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rotary", [True, False])
@pytest.mark.parametrize("paged", [False, True])
def test_vector_path(H, B, S, past, dtype, rotary, paged):
    from onnxruntime_b200.ops import _kernels as K
    N, Nk, T = 6, 2, 256
    g = torch.Generator(device="cuda").manual_seed(H + S)
    qkv = torch.randn(B, S, (N + 2 * Nk) * H, generator=g, device="cuda").to(dtype)
    angle = torch.rand(T, H // 2, generator=g, device="cuda") * 6.28
    cos, sin = (angle.cos().to(dtype), angle.sin().to(dtype)) if rotary else (None, None)
    lens = torch.full((B,), past + S, dtype=torch.int32, device="cuda")

    def run(make):
        shape = (B * 2, 128, Nk, H) if paged else (B, Nk, T, H)
        kc, vc = make(torch.zeros(shape, dtype=dtype, device="cuda")), make(torch.zeros(shape, dtype=dtype, device="cuda"))
        c, s = (make(cos), make(sin)) if rotary else (None, None)
        if not paged:
            q = K.gqa_prep(make(qkv), kc, vc, lens - 1, c, s, N, Nk, H, first_prompt=past == 0)
            return q, kc[:, :, past:past + S].transpose(1, 2), vc[:, :, past:past + S].transpose(1, 2)
        cu = torch.arange(B + 1, dtype=torch.int32, device="cuda") * S
        table = torch.arange(2 * B, dtype=torch.int32, device="cuda").view(B, 2)
        q = K.paged_prep(make(qkv.view(B * S, -1)), kc, vc, cu, lens - S, table, N, Nk, c, s)
        return q.view(B, S, N, H), kc.view(B, T, Nk, H)[:, past:past + S], vc.view(B, T, Nk, H)[:, past:past + S]
    got, general = run(lambda t: t.clone()), run(_shifted)
    x = qkv.view(B, S, N + 2 * Nk, H).float()
    if rotary:
        c, s = (t[past:past + S].float()[None, :, None] for t in (cos, sin))
        a, b = x[:, :, :N + Nk].chunk(2, -1)
        x = torch.cat([torch.cat([a * c - b * s, b * c + a * s], -1), x[:, :, N + Nk:]], 2)
    for y, z, r in zip(got, general, (x[:, :, :N], x[:, :, N:N + Nk], x[:, :, N + Nk:])):
        assert torch.equal(y, z)
        # two fp32 products rounded (2^-24 each of at most 6), then 16 bits
        assert ((y.float() - r).abs() <= r.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + 2.0 ** -20).all()
