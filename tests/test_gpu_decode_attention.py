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


def _rotate(x, cos, sin):
    a, b = x.float().chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1).to(x.dtype)


def _decode_case(dtype, N, Nk, totals, capacity, block, fused, splits=0, algo=2, sink=False, softcap=0.0, window=-1, H=128, seed=0):
    """One call with NaN behind every length, against the oracle; with `fused` the new token comes packed and is rotated and appended."""
    from onnxruntime_b200.ops import _kernels as K
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    B = len(totals)
    assert 1 <= min(totals) and max(totals) <= capacity
    lens = torch.tensor(totals, dtype=torch.int32, device="cuda")
    kc, vc = rand(B, capacity, Nk, H), rand(B, capacity, Nk, H)
    behind = torch.arange(capacity, device="cuda")[None] >= (lens - (1 if fused else 0))[:, None]
    kc[behind], vc[behind] = float("nan"), float("nan")
    table = None
    if block:
        table = torch.randperm(B * capacity // block, generator=torch.Generator().manual_seed(seed)).reshape(B, -1).to(torch.int32).cuda()
        k_dev, v_dev = (torch.empty_like(c).view(-1, block, Nk, H) for c in (kc, vc))
        for c, d in ((kc, k_dev), (vc, v_dev)):
            d[table.view(-1).long()] = c.view(-1, block, Nk, H)
    else:
        k_dev, v_dev = (c.transpose(1, 2).contiguous() for c in (kc, vc))
    head_sink = rand(N) if sink else None
    args = dict(splits=splits, block_table=table, head_sink=head_sink, softcap=softcap, window=window, algo=algo)
    if fused:
        qkv = rand(B, (N + 2 * Nk) * H)
        angle = torch.rand(capacity, H // 2, generator=g, device="cuda") * 6.28
        cos, sin = angle.cos().to(dtype), angle.sin().to(dtype)
        out = K.gqa_decode(None, k_dev, v_dev, lens - 1, qkv=qkv, num_heads=N, cos=cos, sin=sin, **args)
        parts = qkv.view(B, N + 2 * Nk, H)
        c, s = (t[(lens - 1).long()].float()[:, None] for t in (cos, sin))
        q, new_k, new_v = _rotate(parts[:, :N], c, s), _rotate(parts[:, N:N + Nk], c, s), parts[:, N + Nk:]
        rows = torch.arange(B, device="cuda"), (lens - 1).long()
        kc[rows], vc[rows] = new_k, new_v
        if block:
            held = [d[table.long()].reshape(B, capacity, Nk, H)[rows] for d in (k_dev, v_dev)]
        else:
            held = [d.transpose(1, 2)[rows] for d in (k_dev, v_dev)]
        # the same two fp32 products and a rounding; the products may be fused
        assert (held[0].float() - new_k.float()).abs().max() <= 2.0 ** (-7 if dtype == torch.bfloat16 else -10) * float(new_k.float().abs().max())
        assert torch.equal(held[1], new_v)
    else:
        q = rand(B, N, H)
        out = K.gqa_decode(q, k_dev, v_dev, lens - 1, **args)
    limit = vc[~behind]
    for b, total in enumerate(totals):
        first = max(0, total - window) if window > 0 else 0
        _close(out.view(B, N, H)[b], _oracle(q[b], kc[b], vc[b], total, first, head_sink, softcap), limit, dtype)


TILES = [1, 100, 128, 129, 200, 256, 257, 300, 384, 385, 512, 513, 640, 700, 768, 769, 895, 896, 897, 1000]   # one to eight tiles of 128


@pytest.mark.parametrize("block", [0, 16, 256])
@pytest.mark.parametrize("group", [4, 8, 16])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_grids_beyond_the_machine(block, group, fused, dtype):
    """More CTAs than SMs: K and V share three slots a CTA."""
    _decode_case(dtype, 8 * group, 8, TILES, 1024, block, fused, splits=1, seed=group)


@pytest.mark.parametrize("options", [dict(), dict(sink=True), dict(softcap=20.0), dict(sink=True, softcap=20.0)])
@pytest.mark.parametrize("block", [0, 64])
@pytest.mark.parametrize("fused", [False, True])
def test_grids_beyond_the_machine_with_options(options, block, fused):
    _decode_case(torch.bfloat16, 32, 8, TILES, 1024, block, fused, splits=1, seed=5, **options)
    _decode_case(torch.bfloat16, 32, 8, TILES, 1024, block, fused, splits=3, seed=6, **options)


@pytest.mark.parametrize("window", [1, 127, 128, 300])
@pytest.mark.parametrize("fused", [False, True])
def test_grids_beyond_the_machine_with_a_window(window, fused):
    for splits in (0, 1, 3):
        _decode_case(torch.bfloat16, 32, 8, TILES, 4096, 0, fused, splits=splits, window=window, seed=window)


@pytest.mark.parametrize("B,capacity,block", [(10, 2560, 256), (10, 4096, 16), (20, 4096, 256), (20, 4096, 0), (12, 8192, 256), (48, 2560, 256)])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("sink", [False, True])
def test_a_sequence_takes_the_splits_that_its_length_needs(B, capacity, block, fused, sink):
    """Large grids with room for long sequences: lengths around the borders between one, two and three splits (2 tiles a split for
    20 sequences of 8 kv heads and fewer, 6 for 48, whose first splits come first)."""
    unit = 768 if B == 48 else 256
    edges = [1, capacity] + [n * unit + d for n in (1, 2, 3) for d in (-1, 0, 1)] + [4 * unit, capacity - 1, capacity - 127, capacity - 128,
                                                                                     capacity // 2, 129, 128, 700, 2000]
    totals = [min(n, capacity) for n in (edges * 4)[:B]]
    _decode_case(torch.bfloat16, 32, 8, totals, capacity, block, fused, sink=sink, seed=B)


@pytest.mark.parametrize("H,algo", [(64, 1), (128, 1), (128, 2)])
@pytest.mark.parametrize("splits", [8, 9, 16, 17, 32])
@pytest.mark.parametrize("sink", [False, True])
def test_many_splits(H, algo, splits, sink):
    """The merge fetches eight splits at a time."""
    _decode_case(torch.bfloat16, 8, 2, [1, 31, 33, 700, 1024], 1024, 0, False, splits=splits, algo=algo, sink=sink, H=H, seed=splits)
    _decode_case(torch.float16, 8, 2, [1, 31, 33, 700, 1024], 1024, 0, True, splits=splits, algo=algo, sink=sink, H=H, seed=splits)
