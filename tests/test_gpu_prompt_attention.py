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


NAN = float("nan")


@pytest.mark.parametrize("N,Nk,H", [(4, 4, 64), (8, 2, 128)])
@pytest.mark.parametrize("S,total", [(1, 1), (64, 64), (63, 63), (70, 129), (130, 190), (5, 193)])
def test_rows_behind_the_last_key_do_not_matter(N, Nk, H, S, total):
    from onnxruntime_b200.ops import _kernels as K
    dtype = torch.bfloat16 if H == 128 else torch.float16
    g = torch.Generator(device="cuda").manual_seed(N * 100 + S)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    B, T = 2, 256
    q, k, v = rand(B, S, N, H), rand(B, Nk, T, H), rand(B, Nk, T, H)
    lens = torch.tensor([total, total + 3], dtype=torch.int32, device="cuda")
    for b in range(B):
        k[b, :, int(lens[b]):] = NAN
        v[b, :, int(lens[b]):] = NAN
    out = K.attn_prefill(q, k, v, lens - 1, first_prompt=False)
    for b in range(B):
        n = int(lens[b])
        visible = torch.arange(n, device="cuda") <= (n - S + torch.arange(S, device="cuda"))[:, None]
        _close(out[b], _oracle(q[b], k[b, :, :n].transpose(0, 1), v[b, :, :n].transpose(0, 1), visible, H ** -0.5), v[b, :, :n], dtype)


@pytest.mark.parametrize("keys", [1, 63, 64, 65, 200])
def test_rows_behind_the_last_unmasked_key_do_not_matter(keys):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(keys)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").half()  # noqa: E731
    B, S, T, N, H = 2, 130, 260, 2, 64
    q, k, v = rand(B, S, N, H), rand(B, T, N, H), rand(B, T, N, H)
    k[:, keys:], v[:, keys:] = NAN, NAN
    mask = (torch.arange(T, device="cuda") < keys).to(torch.int32).repeat(B, 1)
    out = K.attn_prefill(q, k, v, None, first_prompt=True, causal=False, kv_layout="bsnh", key_mask=mask)
    for b in range(B):
        _close(out[b], _oracle(q[b], k[b, :keys], v[b, :keys], torch.ones(S, keys, dtype=torch.bool, device="cuda"), H ** -0.5), v[b, :keys], torch.float16)


@pytest.mark.parametrize("split_weights", [False, True])
@pytest.mark.parametrize("N,Nk,H", [(8, 2, 128), (4, 4, 64), (8, 1, 128)])
def test_rows_behind_a_packed_sequence_do_not_matter(N, Nk, H, split_weights):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(N)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    batch, bs, blocks = [(0, 1), (0, 130), (127, 1), (300, 33), (64, 64), (511, 1), (5, 16)], 128, 5
    cu = torch.tensor([0] + torch.tensor([n for _, n in batch]).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    past = torch.tensor([p for p, _ in batch], dtype=torch.int32, device="cuda")
    table = torch.randperm(len(batch) * blocks, generator=torch.Generator().manual_seed(1)).reshape(len(batch), blocks).to(torch.int32).cuda()
    q = rand(int(cu[-1]), N, H)
    kc, vc = (torch.full((len(batch) * blocks, bs, Nk, H), NAN, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    rows = []
    for b, (p, n) in enumerate(batch):
        k, v = rand(p + n, Nk, H), rand(p + n, Nk, H)
        rows.append((k, v))
        for c, x in ((kc, k), (vc, v)):
            whole = c[table[b].long()].reshape(-1, Nk, H)
            whole[:p + n] = x
            c[table[b].long()] = whole.reshape(blocks, bs, Nk, H)
    out = K.attn_prefill_paged(q, kc, vc, cu, past, table, split_weights=split_weights)
    for b, (p, n) in enumerate(batch):
        visible = torch.arange(p + n, device="cuda") <= (p + torch.arange(n, device="cuda"))[:, None]
        _close(out[int(cu[b]):int(cu[b + 1])], _oracle(q[int(cu[b]):int(cu[b + 1])], *rows[b], visible, H ** -0.5), rows[b][1], torch.bfloat16)


def test_packed_latent_prompts_do_not_meet():
    """Expanded keys and values lie sequence behind sequence: what one holds must not reach another."""
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    N, dk, dr, dv, lens, past = 4, 32, 16, 32, [70, 1, 33], [5, 60, 0]
    rows = [n + p for n, p in zip(lens, past)]
    T, cols = sum(lens), N * (dk + dr) + N
    x, q_rot, kv, kr, sink = rand(T, cols + -cols % 8), rand(T, N, dr), rand(sum(rows), N * (dk + dv)), rand(sum(rows), dr), rand(N)
    cu = torch.tensor([0, 70, 71, 104], dtype=torch.int32, device="cuda")
    run = lambda values: K.latent_prefill(x, q_rot, values, kr, sink, x[:, cols - N:], cu, torch.tensor(past, dtype=torch.int32, device="cuda"),  # noqa: E731
                                          N, dk, dr, dv, 0.15)
    clean = run(kv)
    dirty = kv.clone()
    dirty[rows[0]:rows[0] + rows[1]] = NAN
    out = run(dirty)
    assert torch.isfinite(clean.float()).all()
    assert torch.equal(out[:70], clean[:70]) and torch.equal(out[71:], clean[71:])


@pytest.mark.parametrize("N,rank,dr,bs", [(16, 512, 64, 128), (40, 136, 16, 64), (3, 64, 8, 8)])
def test_rows_behind_a_latent_cache_do_not_matter(N, rank, dr, bs):
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(N)
    lens = torch.tensor([900, 33, 1, 129, 640], dtype=torch.int32, device="cuda")
    B, per = 5, -(-900 // bs)
    table = torch.arange(B * per, dtype=torch.int32, device="cuda").reshape(B, per)
    q = (0.3 * torch.randn(B, N, rank + dr, generator=g, device="cuda")).to(torch.bfloat16)
    cache = torch.randn(B, per * bs, rank + dr, generator=g, device="cuda").to(torch.bfloat16)
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    outs = []
    for fill in (0.0, NAN):
        for b in range(B):
            cache[b, int(lens[b]):] = fill
        outs.append(K.latent_decode(q, cache.view(B * per, bs, -1), cu, lens - 1, table, rank, 0.3))
    assert torch.isfinite(outs[0][0]).all()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
