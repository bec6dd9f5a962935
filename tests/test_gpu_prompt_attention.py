"""Prompt attention: query heads that share a key head as rows of one tile, lengths at the edges of query and key tiles, key masks
(kept as bits up to 8192 keys, whole tiles behind the last visible key left out), single tokens among prompts."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(q, k, v, visible, scale):
    """q [S, N, H], k / v [T, Nk, H], visible bool [S, T]; a row that sees nothing gives 0."""
    group = q.shape[1] // k.shape[1]
    k, v = (t.double().repeat_interleave(group, 1) for t in (k, v))
    s = torch.einsum("snh,tnh->nst", q.double(), k) * scale
    s = s.masked_fill(~visible, -math.inf)
    p = torch.nan_to_num(s.softmax(-1), nan=0.0)
    return torch.einsum("nst,tnh->snh", p, v)


def _close(y, z, v, dtype):
    # the weights (their sum is 1) and the result are rounded to 16 bits once each; scores differ by fp32 sums (2^-18 of |s| < 32)
    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    assert (y.double() - z).abs().max() <= (2.1 * unit + 2.0 ** -13) * float(v.abs().max())


@pytest.mark.parametrize("N,Nk", [(4, 4), (6, 2), (8, 4), (8, 2), (8, 1), (16, 1)])
@pytest.mark.parametrize("H,S,past", [(64, 1, 0), (64, 129, 0), (64, 40, 88), (128, 63, 1), (128, 64, 0), (128, 257, 70), (128, 9, 247)])
def test_grouped_heads_causal(N, Nk, H, S, past):
    from onnxruntime_b200.ops import _kernels as K
    dtype = torch.bfloat16 if H == 128 else torch.float16
    g = torch.Generator(device="cuda").manual_seed(N * 100 + S)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    B, T = 2, past + S + 5
    q, k, v = rand(B, S, N, H), rand(B, Nk, T, H), rand(B, Nk, T, H)
    lens = torch.full((B,), past + S - 1, dtype=torch.int32, device="cuda")
    out = K.attn_prefill(q, k, v, lens, first_prompt=past == 0)
    visible = torch.arange(T, device="cuda") <= (past + torch.arange(S, device="cuda"))[:, None]
    for b in range(B):
        _close(out[b], _oracle(q[b], k[b].transpose(0, 1), v[b].transpose(0, 1), visible, H ** -0.5), v, dtype)


@pytest.mark.parametrize("T", [1, 64, 65, 200, 384, 8192, 8200])
def test_key_masks(T):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").half()  # noqa: E731
    B, S, N, H = 4, 130, 2, 64
    q, k, v = rand(B, S, N, H), rand(B, T, N, H), rand(B, T, N, H)
    mask = (torch.rand(B, T, generator=g, device="cuda") < 0.5).to(torch.int32)
    mask[1] = torch.arange(T, device="cuda") <= T // 2     # right-padded
    mask[2] = 0                                            # nothing to see
    mask[3] = torch.arange(T, device="cuda") == T - 1
    out = K.attn_prefill(q, k, v, None, first_prompt=True, causal=False, kv_layout="bsnh", key_mask=mask)
    for b in range(B):
        _close(out[b], _oracle(q[b], k[b], v[b], (mask[b] != 0).expand(S, T), H ** -0.5), v, torch.float16)


@pytest.mark.parametrize("N,Nk,H", [(8, 2, 128), (4, 4, 64), (16, 2, 128)])
def test_packed_prompts_and_single_tokens(N, Nk, H):
    from onnxruntime_b200.ops import _kernels as K
    dtype = torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(N)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    batch = [(0, 1), (0, 130), (127, 1), (300, 33), (64, 64), (511, 1), (5, 16)]
    bs, blocks = 128, 5
    cu = torch.tensor([0] + torch.tensor([n for _, n in batch]).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    past = torch.tensor([p for p, _ in batch], dtype=torch.int32, device="cuda")
    table = torch.randperm(len(batch) * blocks, generator=torch.Generator().manual_seed(1)).reshape(len(batch), blocks).to(torch.int32).cuda()
    q, kc, vc = rand(int(cu[-1]), N, H), rand(len(batch) * blocks, bs, Nk, H), rand(len(batch) * blocks, bs, Nk, H)
    out = K.attn_prefill_paged(q, kc, vc, cu, past, table)
    for b, (p, n) in enumerate(batch):
        k, v = (c[table[b].long()].reshape(-1, Nk, H)[:p + n] for c in (kc, vc))
        visible = torch.arange(p + n, device="cuda") <= (p + torch.arange(n, device="cuda"))[:, None]
        _close(out[int(cu[b]):int(cu[b + 1])], _oracle(q[int(cu[b]):int(cu[b + 1])], k, v, visible, H ** -0.5), vc, dtype)
