"""What the speed of this framework is measured on: the GPU configurations that its benchmarks quote, each over the sizes that it serves.

Four kinds of work, all through the session API:

* ``decode`` / ``prefill``: a Llama-shaped decoder with contiguous caches behind ``DecoderRunner`` (8B widths, 8 or 4 of its 32 layers, which are all
  alike, and the whole vocabulary), one captured decode step or one eager prompt;
* ``paged``: the serving form of the decoder (PagedAttention, blocks of 256 tokens) with caches that the caller owns, bound through ``IOBinding``:
  one token for each of many sequences of unequal length (captured), or a batch that mixes new prompts, portions of prompts and single tokens (eager);
  dense bf16 at 8B widths, or 4-bit MatMulNBits in fp16 at 70B widths (4 of its 80 layers);
* ``bert``: a BERT-large-shaped encoder over right-padded batches: 8 of its 24 layers in fp16 from the exporter-style graph, or 2 in fp8 (GemmFloat8: a
  value next to an e4m3 rounding border lands on either side of it, and more layers would multiply that beyond what can be compared);
* ``moe``: one Mixtral-shaped mixture-of-experts layer (bf16, top 2 of 8).

Weights and inputs are random, made from the seed on the GPU.
"""
import math
import random

import numpy as np
import torch

VOCAB, BLOCK = 128256, 256
WIDTHS = {"8b": dict(hidden=4096, heads=32, kv=8, ffn=14336), "70b": dict(hidden=8192, heads=64, kv=8, ffn=28672)}
HEAD = 128
BERT = dict(hidden=1024, heads=16, ffn=4096, vocab=30522, positions=512)
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ------------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one user at a chat: a step is nothing but latency and the stream of weights
        dict(name="decode_1x211", kind="decode", dtype="bf16", layers=8, batch=1, context=211),
        # the headline configuration: batch 8 behind a prompt of 1024
        dict(name="decode_8x1024", kind="decode", dtype="bf16", layers=8, batch=8, context=1024),
        # a serving batch: 40 sequences of unequal length up to 4000 tokens over one pool of blocks
        dict(name="paged_decode_40x4000", kind="paged", model="8b", bits=16, dtype="bf16", layers=8, prompts=0, portions=0, singles=40, context=4000, new=0),
        # 4-bit weights at 4096 tokens of context, one sequence and a batch of 32
        dict(name="int4_decode_1x4096", kind="paged", model="70b", bits=4, dtype="fp16", layers=4, prompts=0, portions=0, singles=1, context=4096, new=0),
        dict(name="int4_decode_32x4096", kind="paged", model="70b", bits=4, dtype="fp16", layers=4, prompts=0, portions=0, singles=32, context=4096, new=0),
        # a short question: time to the first token of 37 tokens
        dict(name="prefill_1x37", kind="prefill", dtype="bf16", layers=4, batch=1, seq=37),
        # the headline configuration's prompt run, the largest call
        dict(name="prefill_8x1024", kind="prefill", dtype="bf16", layers=4, batch=8, seq=1024),
        # a serving step that admits three prompts and continues two others while 20 sequences decode
        dict(name="paged_mixed_2k", kind="paged", model="8b", bits=16, dtype="bf16", layers=4, prompts=3, portions=2, singles=20, context=1500, new=700),
        # encoder: one sentence, and the throughput configuration
        dict(name="bert_1x27", kind="bert", dtype="fp16", layers=8, batch=1, seq=27),
        dict(name="bert_64x384", kind="bert", dtype="fp16", layers=8, batch=64, seq=384),
        # the 8-bit encoder, a mid-sized batch of odd length
        dict(name="bert_fp8_24x317", kind="bert", dtype="fp8", layers=2, batch=24, seq=317),
        # mixture of experts: the prompt configuration (16 x 512 tokens); drawn cases go down to one token
        dict(name="moe_8192", kind="moe", tokens=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "paged_decode", "int4_decode", "prefill", "mixed", "int4_mixed", "bert", "bert_fp8", "moe"])
    if kind == "decode":
        batch = _log(rng, 1, 48)
        return dict(kind="decode", dtype=rng.choice(["bf16", "fp16"]), layers=8, batch=batch, context=_log(rng, 16, min(8000, 130000 // batch)))
    if kind == "paged_decode":
        return dict(kind="paged", model="8b", bits=16, dtype=rng.choice(["bf16", "fp16"]), layers=8, prompts=0, portions=0, singles=_log(rng, 1, 64), context=_log(rng, 40, 4000), new=0)
    if kind == "int4_decode":
        model = rng.choice(["8b", "70b"])
        return dict(kind="paged", model=model, bits=4, dtype=rng.choice(["bf16", "fp16"]), layers=4, prompts=0, portions=0, singles=_log(rng, 1, 48), context=_log(rng, 40, 4096), new=0)
    if kind == "prefill":
        batch = _log(rng, 1, 16)
        return dict(kind="prefill", dtype=rng.choice(["bf16", "fp16"]), layers=4, batch=batch, seq=_log(rng, 5, min(4000, 6500 // batch)))
    if kind in ("mixed", "int4_mixed"):
        return dict(kind="paged", model="8b", bits=4 if kind == "int4_mixed" else 16, dtype=rng.choice(["bf16", "fp16"]), layers=4,
                    prompts=rng.randint(1, 4), portions=rng.randint(0, 3), singles=rng.randint(0, 30), context=_log(rng, 40, 3000), new=_log(rng, 12, 900))
    if kind in ("bert", "bert_fp8"):
        seq = _log(rng, 8, 512)
        return dict(kind="bert", dtype="fp8" if kind == "bert_fp8" else "fp16", layers=2 if kind == "bert_fp8" else 8, batch=_log(rng, 1, min(64, 24000 // seq)), seq=seq)
    return dict(kind="moe", tokens=_log(rng, 1, 8000))


# ---------------------------------------------------------------------------------------------------------- shapes of a case
def _entries(case):
    """[(tokens in the cache, new tokens)] of a paged batch.  The lengths belong to the case and not to the seed."""
    r = random.Random("%(prompts)d/%(portions)d/%(singles)d/%(context)d/%(new)d" % case)
    upto = lambda n: r.randint(max(1, n // 4), max(1, n))  # noqa: E731
    got = [(0, upto(case["new"])) for _ in range(case["prompts"])]
    got += [(upto(case["context"]), upto(case["new"])) for _ in range(case["portions"])]
    return got + [(upto(case["context"]), 1) for _ in range(case["singles"])]


def _capacity(tokens):
    return (tokens + BLOCK - 1) // BLOCK * BLOCK


def _decoder_batch(case):
    if case["kind"] == "paged":
        return _entries(case)
    return [(case["context"], 1) if case["kind"] == "decode" else (0, case["seq"])] * case["batch"]


def work(case):
    if case["kind"] == "moe":
        t, h, f = case["tokens"], 4096, 14336
        experts = min(8, 8 * (1 - 0.75 ** t))     # experts that a batch of t tokens reaches on average
        return {"bytes": 2 * (experts * 3 * h * f + 2 * t * h + 8 * t), "flops": t * 2 * 6 * h * f}
    if case["kind"] == "bert":
        h, f, t = BERT["hidden"], BERT["ffn"], case["batch"] * case["seq"]
        size = 1 if case["dtype"] == "fp8" else 2
        return {"bytes": case["layers"] * size * (4 * h * h + 2 * h * f) + 2 * 2 * t * h + 16 * t,
                "flops": case["layers"] * t * (8 * h * h + 4 * h * f + 4 * case["seq"] * h)}
    w = WIDTHS[case.get("model", "8b")]
    batch = _decoder_batch(case)
    tokens, rows = sum(n for _, n in batch), len(batch)
    cached = sum(p for p, _ in batch)
    matrix = w["hidden"] * (w["heads"] + 2 * w["kv"]) * HEAD + w["heads"] * HEAD * w["hidden"] + 3 * w["hidden"] * w["ffn"]
    weight_bytes = 0.5 + 2 / 32 if case.get("bits") == 4 else 2
    kv = 2 * w["kv"] * HEAD * 2
    pairs = sum(p * n + n * (n + 1) // 2 for p, n in batch)
    return {"bytes": case["layers"] * (matrix * weight_bytes + (cached + tokens) * kv) + 2 * VOCAB * w["hidden"] + 2 * rows * VOCAB + 2 * tokens * w["hidden"],
            "flops": case["layers"] * (2 * tokens * matrix + 4 * w["heads"] * HEAD * pairs) + 2 * rows * VOCAB * w["hidden"]}


def tolerance(case):
    """Four times what the outputs are off from 64-bit sums (see ``exact``: 0.0039 for the mixture of experts, 0.001 and 0.0025 for the fp16 encoder and
    decoder), and the most that can be stated where that is over 0.03 (bf16 hidden states through the layers: 0.014 to 0.023; e4m3: 0.018 to 0.024)."""
    if case["kind"] == "moe":
        return {"rel": 0.015, "max": 0.15}
    if case["kind"] == "bert":
        return {"rel": 0.03, "max": 0.6} if case["dtype"] == "fp8" else {"rel": 0.004, "max": 0.2}
    return {"rel": 0.03, "max": 0.5} if case["dtype"] == "bf16" else {"rel": 0.01, "max": 0.2}


# ------------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _normal(gen, shape, dtype, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0, std, generator=gen)


def _llama(case, seed):
    from onnxruntime_b200.models.llama import LlamaConfig, build_llama
    w = WIDTHS[case.get("model", "8b")]
    longest = _capacity(max(p + n for p, n in _decoder_batch(case)))
    cfg = LlamaConfig(vocab_size=VOCAB, hidden_size=w["hidden"], num_layers=case["layers"], num_heads=w["heads"], num_kv_heads=w["kv"], head_dim=HEAD,
                      ffn_size=w["ffn"], max_seq_len=longest, dtype=case["dtype"])
    model, weights = build_llama(cfg, external_weights=True, seed=int(seed) % 1000003, device="cuda", quant_bits=4 if case.get("bits") == 4 else 0,
                                 paged=case["kind"] == "paged")
    g = _gen(seed, 6)
    for n, q in weights.items():
        if n.endswith(".q4"):    # nibbles 1 to 15 around the zero point 8: like a checkpoint's weights, without a common offset
            q.copy_(torch.randint(1, 16, q.shape, generator=g, device="cuda", dtype=torch.uint8) + 16 * torch.randint(1, 16, q.shape, generator=g, device="cuda", dtype=torch.uint8))
    return cfg, model, weights


def _contiguous_caches(case, seed, layers):
    """Keys and values of the context, [batch, kv heads, context, head] per layer: what an earlier prompt left behind."""
    g = _gen(seed, 2)
    shape = (case["batch"], WIDTHS["8b"]["kv"], case["context"], HEAD)
    return [(_normal(g, shape, DTYPES[case["dtype"]]), _normal(g, shape, DTYPES[case["dtype"]])) for _ in range(layers)]


def _paged_inputs(case, seed):
    g, entries = _gen(seed, 3), _entries(case)
    w, dt = WIDTHS[case["model"]], DTYPES[case["dtype"]]
    needed = [_capacity(p + n) // BLOCK for p, n in entries]
    order = torch.randperm(sum(needed), generator=g, device="cuda").to(torch.int32).split(needed)
    table = torch.zeros(len(entries), max(needed), dtype=torch.int32, device="cuda")
    for b, blocks in enumerate(order):
        table[b, :len(blocks)] = blocks
    ends = np.cumsum([n for _, n in entries])
    device = lambda v, dt: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    inputs = {"input_ids": torch.randint(0, VOCAB, (int(ends[-1]),), generator=g, device="cuda"), "block_table": table,
              "cumulative_sequence_length": device([0] + ends.tolist(), torch.int32), "past_seqlens": device([p for p, _ in entries], torch.int32),
              "logits_indices": device((ends - 1).tolist(), torch.int64)}
    shape = (sum(needed), BLOCK, w["kv"], HEAD)
    caches = {"%s_cache.%d" % (kv, i): _normal(g, shape, dt) for i in range(case["layers"]) for kv in ("key", "value")}
    return inputs, caches


def _bert(case, seed):
    g, h, f = _gen(seed, 4), BERT["hidden"], BERT["ffn"]
    shapes = {"embeddings.word": (BERT["vocab"], h), "embeddings.position": (BERT["positions"], h)}
    for i in range(case["layers"]):
        p = "layer.%d." % i
        shapes.update({p + "attn.%s.weight" % n: (h, h) for n in "qkvo"})
        shapes.update({p + "attn.%s.bias" % n: (h,) for n in "qkvo"})
        shapes.update({p + "ffn.fc1.weight": (h, f), p + "ffn.fc1.bias": (f,), p + "ffn.fc2.weight": (f, h), p + "ffn.fc2.bias": (h,)})
    w = {n: _normal(g, s, torch.float16, 0.02) for n, s in shapes.items()}
    for n in ["embeddings.ln"] + ["layer.%d.%s.ln" % (i, b) for i in range(case["layers"]) for b in ("attn", "ffn")]:
        w[n + ".gamma"], w[n + ".beta"] = torch.ones(h, dtype=torch.float16, device="cuda"), torch.zeros(h, dtype=torch.float16, device="cuda")
    ids = torch.randint(0, BERT["vocab"], (case["batch"], case["seq"]), generator=g, device="cuda")
    lengths = torch.randint(max(1, case["seq"] // 2), case["seq"] + 1, (case["batch"], 1), generator=g, device="cuda")
    return w, ids, (torch.arange(case["seq"], device="cuda") < lengths).to(torch.int64)


def _moe(case, seed):
    g, h, f = _gen(seed, 5), 4096, 14336
    bf16 = torch.bfloat16
    return {"x": _normal(g, (case["tokens"], h), bf16, 0.5), "router": _normal(g, (case["tokens"], 8), bf16),
            "fc1": _normal(g, (8, f, h), bf16, 0.02), "fc2": _normal(g, (8, h, f), bf16, 0.02), "fc3": _normal(g, (8, f, h), bf16, 0.02)}


# ------------------------------------------------------------------------------------------------------------ prepare and run
def _session(model, weights=None, graph=False):
    import onnxruntime_b200 as ort
    so = ort.SessionOptions()
    if weights:
        so.add_external_initializers(list(weights), list(weights.values()))
    return ort.InferenceSession(model, so, providers=[("CUDAExecutionProvider", {"device_id": "0", "enable_cuda_graph": "1" if graph else "0"})], enable_fallback=False)


def prepare(case, seed):
    import onnxruntime_b200 as ort
    from onnxruntime_b200 import onnx_lite as ol
    from onnxruntime_b200.models.bert import BertConfig, build_bert, build_bert_fp8
    from onnxruntime_b200.models.generation import DecoderRunner
    if case["kind"] == "bert":
        w, ids, mask = _bert(case, seed)
        cfg = BertConfig.bert_large(num_layers=case["layers"])
        sess = _session((build_bert_fp8 if case["dtype"] == "fp8" else build_bert)(cfg, {n: t.cpu().numpy() for n, t in w.items()}))
        out = torch.empty(case["batch"], case["seq"], BERT["hidden"], dtype=torch.float16, device="cuda")
        binding = sess.io_binding()
        binding.bind_torch_input("input_ids", ids)
        binding.bind_torch_input("attention_mask", mask)
        binding.bind_torch_output(sess.get_outputs()[0].name, out)
        return dict(case, sess=sess, binding=binding, out=out, options=None)
    if case["kind"] == "moe":
        t, T = _moe(case, seed), ol.TensorProto
        weights = {n: t[n] for n in ("fc1", "fc2", "fc3")}
        node = ol.make_node("MoE", ["x", "router", "fc1", "", "fc2", "", "fc3"], ["y"], domain="com.microsoft", k=2, activation_type="silu", normalize_routing_weights=1)
        info = lambda n, c: ol.make_tensor_value_info(n, T.BFLOAT16, ["tokens", c])  # noqa: E731
        graph = ol.make_graph([node], "moe", [info("x", 4096), info("router", 8)], [info("y", 4096)],
                              [ol.make_external_tensor(n, T.BFLOAT16, list(w.shape)) for n, w in weights.items()])
        sess = _session(ol.make_model(graph).serialize(), weights)
        out = torch.empty_like(t["x"])
        binding = sess.io_binding()
        binding.bind_torch_input("x", t["x"])
        binding.bind_torch_input("router", t["router"])
        binding.bind_torch_output("y", out)
        return dict(case, sess=sess, binding=binding, out=out, options=None)
    cfg, model, weights = _llama(case, seed)
    if case["kind"] == "paged":
        captured = case["prompts"] + case["portions"] == 0      # one token per sequence: fixed shapes and addresses
        sess = _session(model, weights, graph=captured)
        inputs, caches = _paged_inputs(case, seed)
        logits = torch.empty(len(_entries(case)), VOCAB, dtype=DTYPES[case["dtype"]], device="cuda")
        tokens = torch.empty(len(_entries(case)), dtype=torch.int64, device="cuda")
        binding = sess.io_binding()
        for n, t in list(inputs.items()) + list(caches.items()):
            binding.bind_torch_input(n, t)
        for n, t in caches.items():
            binding.bind_torch_output(n.replace("_cache.", "_cache_out."), t)
        binding.bind_torch_output("logits", logits)
        binding.bind_torch_output("next_tokens", tokens)
        options = ort.RunOptions()
        options.add_run_config_entry("gpu_graph_id", "1" if captured else "-1")
        return dict(case, sess=sess, binding=binding, out=[logits] + list(caches.values()), options=options)
    sess = _session(model, weights, graph=case["kind"] == "decode")
    g = _gen(seed, 1)
    if case["kind"] == "prefill":
        runner = DecoderRunner(sess, cfg, case["batch"], _capacity(case["seq"]))
        return dict(case, runner=runner, ids=torch.randint(0, VOCAB, (case["batch"], case["seq"]), generator=g, device="cuda"))
    runner = DecoderRunner(sess, cfg, case["batch"], _capacity(case["context"] + 1))
    for (k, v), (key, value) in zip(runner.cache, _contiguous_caches(case, seed, case["layers"])):
        k[:, :, :case["context"]], v[:, :, :case["context"]] = key, value
    return dict(case, runner=runner, ids=torch.randint(0, VOCAB, (case["batch"], 1), generator=g, device="cuda"))


def run(state):
    """Logits (or hidden states) and the caches as the pass leaves them; the arg-max, which random weights leave to ties, is computed and not compared."""
    if state["kind"] in ("bert", "moe", "paged"):
        state["sess"].run_with_iobinding(state["binding"], state["options"])
        return state["out"]
    runner = state["runner"]
    if state["kind"] == "prefill":
        runner.prefill(state["ids"])
        return [runner.prefill_logits, runner.cache]
    runner.cur_len = state["context"]
    runner.decode_step(state["ids"])
    return [runner.step_logits, runner.cache]


# -------------------------------------------------------------------------------------------------------------- 64-bit results
def _rms(x, gain, eps=1e-5):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain.double()


def _matrix(weights, name):
    """[in, out] in 64 bits; 4-bit weights: nibble - 8, low nibble first, times the scale of their block of 32 inputs."""
    if name in weights:
        return weights[name].double()
    q, s = weights[name + ".q4"], weights[name + ".scales"].double()
    q = torch.stack([q & 15, q >> 4], -1).reshape(q.shape[0], q.shape[1], -1).double() - 8
    return (q * s.reshape(q.shape[0], q.shape[1], 1)).reshape(q.shape[0], -1).t()


def _exact_llama(case, weights, ids, batch, past):
    """``past(layer, b)``: keys and values [kv heads, tokens, head] of sequence b.  Returns the logits of every last token and [layer][b] new keys and values."""
    w = WIDTHS[case.get("model", "8b")]
    group = w["heads"] // w["kv"]
    x = weights["model.embed_tokens.weight"][ids].double()
    place = torch.cat([torch.arange(p, p + n, device="cuda") for p, n in batch])
    cos, sin = (weights[n][place].double().unsqueeze(1) for n in ("cos_cache", "sin_cache"))
    starts, new = np.cumsum([0] + [n for _, n in batch]).tolist(), []

    def rotate(t):
        a, b = t.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        qkv = (_rms(x, weights[p + "input_layernorm.weight"]) @ _matrix(weights, p + "attn.qkv_proj.weight")).reshape(len(x), -1, HEAD)
        q, k, v = rotate(qkv[:, :w["heads"]]), rotate(qkv[:, w["heads"]:w["heads"] + w["kv"]]), qkv[:, w["heads"] + w["kv"]:]
        ctx, new_i = torch.empty_like(q), []
        for b, (held, n) in enumerate(batch):
            rows = slice(starts[b], starts[b] + n)
            kb, vb = k[rows].transpose(0, 1), v[rows].transpose(0, 1)
            new_i.append((kb, vb))
            pk, pv = past(i, b)
            kb, vb = torch.cat([pk.double(), kb], 1), torch.cat([pv.double(), vb], 1)
            hidden = torch.arange(held + n, device="cuda") > torch.arange(held, held + n, device="cuda").unsqueeze(1)
            for j in range(w["kv"]):
                s = q[rows, j * group:(j + 1) * group].transpose(0, 1) @ kb[j].t() / math.sqrt(HEAD)
                ctx[rows, j * group:(j + 1) * group] = (s.masked_fill_(hidden, -math.inf).softmax(-1) @ vb[j]).transpose(0, 1)
        x = x + ctx.reshape(len(x), -1) @ _matrix(weights, p + "attn.o_proj.weight")
        y = _rms(x, weights[p + "post_attention_layernorm.weight"])
        y = torch.nn.functional.silu(y @ _matrix(weights, p + "mlp.gate_proj.weight")) * (y @ _matrix(weights, p + "mlp.up_proj.weight"))
        x = x + y @ _matrix(weights, p + "mlp.down_proj.weight")
        new.append(new_i)
    return _rms(x[[s - 1 for s in starts[1:]]], weights["model.norm.weight"]) @ weights["lm_head.weight"].double(), new


def _exact_bert(case, w, ids, mask):
    h, n = BERT["hidden"], BERT["heads"]
    f = torch.nn.functional
    norm = lambda t, name: f.layer_norm(t, (h,), w[name + ".gamma"].double(), w[name + ".beta"].double(), 1e-12)  # noqa: E731
    fp8 = case["dtype"] == "fp8"

    def dense(t, name):
        m, bias = w[name + ".weight"].double(), w[name + ".bias"].double()
        if not fp8:
            return t @ m + bias
        scale = float(np.float32(float(w[name + ".weight"].float().abs().max()) / 448.0))
        return (t.to(torch.float16).to(torch.float8_e4m3fn).double() @ (w[name + ".weight"].float() / scale).to(torch.float8_e4m3fn).double()) * scale + bias

    def dense_qkv(t, p):
        names = [p + "attn.%s" % c for c in "qkv"]
        if not fp8:
            return [dense(t, m) for m in names]
        scale = float(np.float32(max(float(w[m + ".weight"].float().abs().max()) for m in names) / 448.0))    # one matrix, one scale
        t = t.to(torch.float16).to(torch.float8_e4m3fn).double()
        return [t @ (w[m + ".weight"].float() / scale).to(torch.float8_e4m3fn).double() * scale + w[m + ".bias"].double() for m in names]
    x = norm(w["embeddings.word"][ids].double() + w["embeddings.position"][:case["seq"]].double(), "embeddings.ln")
    hidden = (mask == 0)[:, None, None, :]
    for i in range(case["layers"]):
        p = "layer.%d." % i
        q, k, v = (t.reshape(*ids.shape, n, h // n).transpose(1, 2) for t in dense_qkv(x, p))
        s = (q @ k.transpose(-1, -2) / math.sqrt(h // n)).masked_fill_(hidden, -math.inf).softmax(-1)
        x = norm(dense((s @ v).transpose(1, 2).reshape(x.shape), p + "attn.o") + x, p + "attn.ln")
        x = norm(dense(f.gelu(dense(x, p + "ffn.fc1")), p + "ffn.fc2") + x, p + "ffn.ln")
    return x


def exact(case, seed):
    if case["kind"] == "bert":
        return _exact_bert(case, *_bert(case, seed))
    if case["kind"] == "moe":
        t = _moe(case, seed)
        share, chosen = t["router"].double().softmax(-1).sort(dim=-1, descending=True, stable=True)
        share, chosen = share[:, :2] / share[:, :2].sum(-1, keepdim=True), chosen[:, :2]
        y = torch.zeros(t["x"].shape, dtype=torch.float64, device="cuda")
        for e in range(8):
            rows, slot = (chosen == e).nonzero(as_tuple=True)
            x = t["x"][rows].double()
            x = torch.nn.functional.silu(x @ t["fc1"][e].double().t()) * (x @ t["fc3"][e].double().t()) @ t["fc2"][e].double().t()
            y[rows] += x * share[rows, slot].unsqueeze(1)
        return y
    _, _, weights = _llama(case, seed)
    batch = _decoder_batch(case)
    if case["kind"] == "paged":
        inputs, caches = _paged_inputs(case, seed)
        table, caches = inputs["block_table"].long(), {n: c.double() for n, c in caches.items()} if sum(c.numel() for c in caches.values()) < 1 << 31 else caches
        places = [(table[b, torch.arange(p + n, device="cuda") // BLOCK], torch.arange(p + n, device="cuda") % BLOCK) for b, (p, n) in enumerate(batch)]

        def past(i, b):
            blocks, rows = (t[:batch[b][0]] for t in places[b])
            return [caches["%s_cache.%d" % (kv, i)][blocks, rows].transpose(0, 1) for kv in ("key", "value")]
        logits, new = _exact_llama(case, weights, inputs["input_ids"], batch, past)
        for i in range(case["layers"]):
            for b, (p, n) in enumerate(batch):
                for j, kv in enumerate(("key", "value")):
                    caches["%s_cache.%d" % (kv, i)][places[b][0][p:], places[b][1][p:]] = new[i][b][j].transpose(0, 1).to(caches["key_cache.0"].dtype)
        return [logits] + list(caches.values())
    decode = case["kind"] == "decode"
    held = _contiguous_caches(case, seed, case["layers"]) if decode else None
    none = torch.empty(WIDTHS["8b"]["kv"], 0, HEAD, dtype=torch.float64, device="cuda")
    ids = torch.randint(0, VOCAB, (case["batch"], 1 if decode else case["seq"]), generator=_gen(seed, 1), device="cuda")
    logits, new = _exact_llama(case, weights, ids.reshape(-1), batch, lambda i, b: [t[b] for t in held[i]] if decode else [none, none])
    capacity, end = _capacity(batch[0][0] + batch[0][1]), batch[0][0] + batch[0][1]
    caches = []
    for i in range(case["layers"]):
        pair = [torch.zeros(case["batch"], WIDTHS["8b"]["kv"], capacity, HEAD, dtype=torch.float64, device="cuda") for _ in range(2)]
        for j in range(2):
            for b in range(case["batch"]):
                if decode:
                    pair[j][b, :, :case["context"]] = held[i][j][b].double()
                pair[j][b, :, batch[b][0]:end] = new[i][b][j]
        caches.append(tuple(pair))
    return [logits.unsqueeze(1), caches]
