"""EmbedLayerNormalization out of Gathers whose positions an exporter derives from the sequence length: the index chain goes,
ids keep Gather's meaning, and sequences beyond the table stay refused."""
import numpy as np
import pytest

import onnxruntime_b200 as ort
from onnxruntime_b200.models.bert import BertConfig, build_bert, init_weights, reference_forward

CPU = ["CPUExecutionProvider"]
CUDA = [("CUDAExecutionProvider", {})]


def _run(providers, ids, segments, max_position=64, hidden=128):
    cfg = BertConfig(type_vocab_size=2 if segments is not None else 0, max_position=max_position, num_layers=1)
    w = init_weights(cfg, 3)
    feeds = {"input_ids": ids, "attention_mask": np.ones_like(ids)}
    if segments is not None:
        feeds["token_type_ids"] = segments
    sess = ort.InferenceSession(build_bert(cfg, w), providers=providers)
    out = sess.run(None, feeds)[0]
    ref = reference_forward(cfg, w, ids % cfg.vocab_size, feeds["attention_mask"], None if segments is None else segments % 2)
    return out, ref


@pytest.mark.parametrize("providers", [CPU, pytest.param(CUDA, marks=pytest.mark.gpu)])
@pytest.mark.parametrize("B,S", [(1, 1), (2, 33), (3, 64)])
@pytest.mark.parametrize("low", [0, -500])
@pytest.mark.parametrize("with_segments", [False, True])
def test_derived_positions(providers, B, S, low, with_segments):
    rng = np.random.RandomState(S)
    ids = rng.randint(low, 1000 + low, (B, S)).astype(np.int64)
    segments = rng.randint(-2 if low else 0, 2, (B, S)).astype(np.int64) if with_segments else None
    out, ref = _run(providers, ids, segments)
    # fp32 layers of width 128; the GPU runs them through 32-bit library products or better
    np.testing.assert_allclose(out, ref, rtol=1e-3, atol=1e-3 if providers is CUDA else 5e-5)


@pytest.mark.parametrize("providers", [CPU, pytest.param(CUDA, marks=pytest.mark.gpu)])
def test_sequence_beyond_the_table_is_refused(providers):
    with pytest.raises(Exception):
        _run(providers, np.zeros((2, 9), np.int64), None, max_position=8)


def test_index_chain_is_gone(tmp_path):
    cfg = BertConfig(num_layers=1)
    so = ort.SessionOptions()
    so.optimized_model_filepath = str(tmp_path / "opt.onnx")
    ort.InferenceSession(build_bert(cfg, init_weights(cfg, 0)), so, providers=CPU)
    from onnxruntime_b200 import onnx_lite as ol
    ops = [n.op_type for n in ol.load_model(so.optimized_model_filepath).graph.nodes]
    assert "EmbedLayerNormalization" in ops and "Slice" not in ops and "Shape" not in ops


@pytest.mark.parametrize("suffix", ["onnx", "ort"])
@pytest.mark.parametrize("providers", [CPU, pytest.param(CUDA, marks=pytest.mark.gpu)])
def test_saved_model_keeps_the_meaning_within_the_schema(tmp_path, providers, suffix):
    """The optimised model has no attribute that the operator's schema lacks, and negative ids mean the same after a reload."""
    from onnxruntime_b200 import onnx_lite as ol, ort_format
    cfg = BertConfig(num_layers=1)
    w = init_weights(cfg, 3)
    so = ort.SessionOptions()
    so.optimized_model_filepath = str(tmp_path / f"opt.{suffix}")
    if suffix == "ort":
        so.add_session_config_entry("session.save_model_format", "ORT")
    first = ort.InferenceSession(build_bert(cfg, w), so, providers=providers)
    with open(so.optimized_model_filepath, "rb") as f:
        saved = f.read()
    assert ort_format.is_ort_format(saved) == (suffix == "ort")
    model = ort_format.ort_to_onnx(saved) if suffix == "ort" else ol.load_model(saved)
    node, = [n for n in model.graph.nodes if n.op_type == "EmbedLayerNormalization"]
    assert {a.name for a in node.attributes} <= {"epsilon", "mask_index_type"}
    assert node.metadata == {"ortb200.from_gathers": "1"}
    ids = np.random.RandomState(0).randint(-500, 500, (2, 9)).astype(np.int64)
    feeds = {"input_ids": ids, "attention_mask": np.ones_like(ids), "token_type_ids": ids % 2 - 2}
    feeds = {k: v for k, v in feeds.items() if k in {i.name for i in first.get_inputs()}}
    again = ort.InferenceSession(so.optimized_model_filepath, providers=providers)
    np.testing.assert_array_equal(first.run(None, feeds)[0], again.run(None, feeds)[0])
    ref = reference_forward(cfg, w, ids % cfg.vocab_size, feeds["attention_mask"], feeds["token_type_ids"] % 2 if "token_type_ids" in feeds else None)
    np.testing.assert_allclose(again.run(None, feeds)[0], ref, rtol=1e-3, atol=1e-3 if providers is CUDA else 5e-5)
