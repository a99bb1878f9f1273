"""The float32 product on the tensor cores (csrc/dense_gemm_split.cuh) at the edges of its tiles: rows around whole tiles of 16 and of 128,
K with partial steps of 32, 64 and 128 elements and split over two and four CTAs, column counts around 128 and around the 64 of the gate/up form.
One-layer Genetar models in float32 against the float64 implementation, held to that mode's 2e-4 of the logits' root mean square, and to 2e-5 of the
CUDA-core kernel's result (both sum up to 1100 f32 products in f32: 1e-6 each, a layer deep).  Option "gemm_split" 1 where the products are too small to take
the kernel by themselves."""
import numpy as np
import pytest

import genetar_oracle as G

pytestmark = pytest.mark.gpu


def model(gpu_lib, tmp_path, width, ff, vocab, seed, change=None):
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=16, vdim=16, ff=ff, v_mix=False)], width=width, vocab=vocab)
    W = G.random_weights(cfg, seed=seed)
    if change:
        change(W)
    return cfg, W, gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=400)


@pytest.mark.parametrize("width,ff,vocab,n", [
    (64, 64, 128, 16), (64, 96, 129, 17), (128, 132, 63, 2), (36, 20, 127, 3), (132, 68, 257, 129), (192, 100, 64, 128), (256, 260, 300, 7),
    (516, 1028, 130, 33), (1100, 192, 65, 113), (260, 512, 128, 400),
])
def test_tile_edges(gpu_lib, tmp_path, width, ff, vocab, n):
    cfg, W, m = model(gpu_lib, tmp_path, width, ff, vocab, width + n)
    toks = np.random.default_rng(n).integers(0, vocab, n).tolist()
    want, _ = G.forward(cfg, W, toks)
    m.set_option("gemm_split", 1)
    got = m.forward_tokens(toks, 0, list(range(n)))
    assert G.rel_rms(got, want) < 2e-4
    m.set_option("gemm_split", 0)
    assert G.rel_rms(got, m.forward_tokens(toks, 0, list(range(n)))) < 2e-5
    m.close()


@pytest.mark.parametrize("what", [np.inf, -np.inf, np.nan, 3e38])
def test_values_beyond_the_pieces(gpu_lib, tmp_path, what):
    """infinities and NaN in a weight, and a sum that leaves f32: the same infinities, NaNs and finite logits as with multiply-adds"""
    def change(W):
        W["head"][5, 3] = what
        W["head"][7, :40] = what
    cfg, _, m = model(gpu_lib, tmp_path, 256, 64, 140, 9, change)
    toks = np.random.default_rng(1).integers(0, 140, 40).tolist()
    m.set_option("gemm_split", 0)
    want = m.forward_tokens(toks, 0, list(range(40)))
    m.set_option("gemm_split", 1)
    got = m.forward_tokens(toks, 0, list(range(40)))
    if np.isfinite(what):   # (a sum of several such terms may or may not leave f32 on the way, by their order: row 7)
        want[:, 7] = got[:, 7] = 0.0
    assert (np.isnan(got) == np.isnan(want)).all() and (np.isposinf(got) == np.isposinf(want)).all() and (np.isneginf(got) == np.isneginf(want)).all()
    assert np.isfinite(what) or not np.isfinite(got[:, [5, 7]]).any()
    both = np.isfinite(want)
    scale = np.where(np.arange(140) == 5, np.abs(what), 1.0) if np.isfinite(what) else 1.0
    got, want = got / scale, want / scale
    assert np.allclose(got[both], want[both], rtol=1e-4, atol=1e-4 * np.abs(np.delete(want, [5, 7], 1)).max())   # (the two kernels' sums: 1e-6)
    m.close()
