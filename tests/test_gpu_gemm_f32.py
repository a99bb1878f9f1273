"""The f32 many-row product (csrc/dense_gemm_f32.cuh) at the edges of its tiles: rows around 64, K with partial 64-element steps (one
or both halves short, less than one step), column counts around 64 and around the 32 of the gate/up form, and a K whose rows do
not start on 16-byte boundaries (the general kernel).  One-layer Genetar models in float32 against the float64 implementation, held to
that mode's 2e-4 of the logits' root mean square.  Its grouped and batched forms run in the Tudatar tests."""
import numpy as np
import pytest

import genetar_oracle as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff,vocab,n", [
    (64, 64, 64, 64), (64, 96, 65, 65), (128, 132, 63, 63), (36, 20, 61, 2), (100, 31, 130, 129), (132, 36, 33, 66), (192, 100, 64, 128),
    (160, 224, 300, 7), (66, 64, 64, 65), (64, 66, 64, 65),
])
def test_tile_edges(gpu_lib, tmp_path, width, ff, vocab, n):
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=16, vdim=16, ff=ff, v_mix=False)], width=width, vocab=vocab)
    W = G.random_weights(cfg, seed=width + n)
    toks = np.random.default_rng(n).integers(0, vocab, n).tolist()
    want, _ = G.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=160)
    assert G.rel_rms(m.forward_tokens(toks, 0, list(range(n))), want) < 2e-4
    m.close()
