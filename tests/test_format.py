"""LMRS v4 format: our layout/quantizer restatement vs files produced by the REFERENCE'S OWN exporter
(tests/golden/*.lmrs, generated by tests/golden/make_golden.py with the reference's export.py)."""
import os

import numpy as np
import pytest

GOLD = os.path.join(os.path.dirname(__file__), "golden")
CASES = ["ref_llama_q8", "ref_gemma_q4", "ref_phi_q8"]


def _load(name):
    return np.fromfile(os.path.join(GOLD, name + ".lmrs"), dtype=np.uint8), np.load(os.path.join(GOLD, name + ".src.npz"))


@pytest.mark.parametrize("name", CASES)
def test_header_and_size_formula(lf, name):
    data, _ = _load(name)
    a = lf.parse_header(data)
    assert a.group_size == 128 and a.multimodal == 0
    assert lf.file_size(a) == data.size                      # 256 + sum of Q(n) / f32 tensors, export.py:87-125
    assert bytes(data[:256]) == a.pack()                     # our header writer == export.py:54-84
    assert not data[55:256].any()


@pytest.mark.parametrize("name", CASES)
def test_tensor_order_and_weight_quantizers(lf, name):
    data, src = _load(name)
    a = lf.parse_header(data)
    offs, end = lf.tensor_offsets(a)
    assert end == data.size
    hf = {"wq": "self_attn.q_proj", "wk": "self_attn.k_proj", "wv": "self_attn.v_proj", "wo": "self_attn.o_proj",
          "w1": "mlp.gate_proj", "w2": "mlp.down_proj", "w3": "mlp.up_proj"}
    quant = lf.quantize_q80 if a.q_type == 1 else lf.quantize_q40
    for l in range(a.n_layers):
        for ours, theirs in hf.items():
            key = f"model.layers.{l}.{theirs}.weight"
            if key in src:
                w = src[key]
            elif ours in ("wq", "wk", "wv"):                  # PHI fused qkv split in thirds (export.py:92-95)
                fused = src[f"model.layers.{l}.self_attn.qkv_proj.weight"]
                third = fused.shape[0] // 3
                w = fused[{"wq": 0, "wk": 1, "wv": 2}[ours] * third:][:third]
            else:                                             # PHI gate_up split in halves (export.py:109-112)
                fused = src[f"model.layers.{l}.mlp.gate_up_proj.weight"]
                half = fused.shape[0] // 2
                w = fused[{"w1": 0, "w3": 1}[ours] * half:][:half]
            q, s = quant(w.reshape(-1), 128)
            qo, so = offs[ours][l]
            assert np.array_equal(data[qo:qo + q.size], q.view(np.uint8)), (ours, l)
            assert np.array_equal(data[so:so + s.size * 4].view(np.float32), s), (ours, l)
        ro = offs["rms_att"][l]
        assert np.array_equal(data[ro:ro + a.dim * 4].view(np.float32), src[f"model.layers.{l}.input_layernorm.weight"])
    q, s = quant(src["model.embed_tokens.weight"].reshape(-1), 128)
    qo, so = offs["emb"][0]
    assert np.array_equal(data[qo:qo + q.size], q.view(np.uint8))
    fo = offs["rms_final"][0]
    assert np.array_equal(data[fo:fo + a.dim * 4].view(np.float32), src["model.norm.weight"])
    if a.model_type == lf.PHI:
        q, s = quant(src["lm_head.weight"].reshape(-1), 128)
        qo, so = offs["lm_head"][0]
        assert np.array_equal(data[qo:qo + q.size], q.view(np.uint8))


@pytest.mark.parametrize("name", CASES)
def test_oracle_loads_reference_files(ref, name):
    data, _ = _load(name)
    m = ref.RefTransformer(data)
    assert m.end_offset == data.size
    lg = m.forward(1, 0)
    assert np.isfinite(lg).all() and lg.shape == (m.args.vocab_size,)


def test_q4_weight_scale_is_minus_7_5_on_disk(lf):
    w = np.array([7.5, -7.5] + [0.0] * 126, np.float32)   # utils/quantization.py:18 (runtime activations use -8)
    q, s = lf.quantize_q40(w, 128)
    assert s[0] == np.float32(-1.0) and q[0] == (0 | (15 << 4)) + 1 - 1   # 7.5/-1+8=0.5 -> round half-even 0; -7.5 -> 15.5 -> 16 -> clamp 15


def test_algorithmic_byte_counts_match_survey(lf):
    assert lf.decode_bytes_per_token(lf.model_args("llama-3.2-1b", 1)) == 1_274_634_240
    assert lf.decode_bytes_per_token(lf.model_args("llama-3.2-3b", 2)) == 1_707_380_736
    assert lf.decode_bytes_per_token(lf.model_args("gemma-2-9b", 1)) == 9_532_307_456
    assert lf.decode_bytes_per_token(lf.model_args("phi-3.5-mini", 1)) == 3_839_502_336
    assert lf.prefill_int8_ops(lf.model_args("llama-3.2-1b", 1), 512) == 2 * 973_078_528 * 512
