"""Decode attention kernels alone, against 64-bit sums: workspaces, grids, splits and cache layouts at their edges."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(q, k, v, total, first=0, sink=None, softcap=0.0):
    """q [N, H], k / v [T, Nk, H]: keys first .. total - 1 of one sequence."""
    group = q.shape[0] // k.shape[1]
    k, v = (t[first:total].double().repeat_interleave(group, 1) for t in (k, v))
    s = torch.einsum("nh,tnh->nt", q.double(), k) / math.sqrt(q.shape[1])
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None]], 1)
    p = s.softmax(-1)[:, :total - first]
    return torch.einsum("nt,tnh->nh", p, v)


def _close(y, z, v, dtype):
    # softmax weights and the result are rounded to 16 bits once each (weights sum to 1); scores are fp32 sums (2^-18 of |s| < 32)
    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    assert (y.double() - z).abs().max() <= (2.1 * unit + 2.0 ** -13) * float(v.double().abs().max())


@pytest.mark.parametrize("H", [64, 128])
@pytest.mark.parametrize("splits", [2, 9])
@pytest.mark.parametrize("offset", [4, 8])
def test_workspace_that_is_aligned_for_floats_only(monkeypatch, H, splits, offset):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(H)
    B, N, Nk, T = 3, 8, 2, 1300
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    q, k, v = rand(B, N, H), rand(B, Nk, T, H), rand(B, Nk, T, H)
    lens = torch.tensor([0, 700, T - 1], dtype=torch.int32, device="cuda")
    need = int(K.lib().ortb200_gqa_decode_workspace_bytes(B, N, H))
    for size in (need + 64, need):      # with room for the padding, and without
        whole = torch.zeros(size + offset, dtype=torch.uint8, device="cuda")
        monkeypatch.setitem(K._ATTN_WS, q.device.index, whole[offset:])
        out = K.gqa_decode(q, k, v, lens, splits=splits).view(B, N, H)
        again = K.gqa_decode(q, k, v, lens, splits=splits).view(B, N, H)     # the counters are left at zero
        assert torch.equal(out, again)
        for b in range(B):
            _close(out[b], _oracle(q[b], k[b].transpose(0, 1), v[b].transpose(0, 1), int(lens[b]) + 1), v, torch.bfloat16)
