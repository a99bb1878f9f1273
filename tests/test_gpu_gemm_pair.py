"""The two-SM tensor-core product (gemm_bf16_pair_kernel) in its three forms -- 256-wide tiles, 128-wide tiles, K split over two pairs --
around whole tiles of 256 rows and of its columns, with partial 64-element steps of K, for the stored, residual and gate/up epilogues.
One-layer Genetar models in bfloat16, every product of more than 128 rows on the form under test (option "gemm_form"; K <= 64 cannot be
split and goes by size) against the same model on the CUDA-core kernel: the two sum in another order, and a sum may round to the
neighbouring bf16 value on the way into the next product (2^-9 of it, here and there)."""
import numpy as np
import pytest

import genetar_oracle as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [-2, -1, 0, 1, 2])
@pytest.mark.parametrize("width,ff,vocab,n", [
    (64, 64, 61, 129),        # few columns, one row in the odd CTA
    (72, 200, 128, 256),      # one whole tile of rows, K that ends inside a step
    (1032, 264, 129, 257),    # 17 steps of K: halves of 8 and 9; one row in the second tile
    (264, 1032, 300, 200),    # the residual product over a longer K than the others
    (1024, 1024, 256, 384),
    (64, 4864, 64, 160),      # gate/up: many column tiles
    (9608, 72, 64, 140),      # residual: many column tiles
    (64, 72, 9700, 130),      # stored logits: many column tiles
    (72, 136, 60, 513),       # three tiles of rows, one row in the last
])
def test_forms_and_edges(gpu_lib, tmp_path, width, ff, vocab, n, form):
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=16, vdim=16, ff=ff, v_mix=False)], width=width, vocab=vocab)
    W = G.random_weights(cfg, seed=width + n)
    toks = np.random.default_rng(n).integers(0, vocab, n).tolist()
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="bfloat16", max_tokens=520)
    m.set_option("gemm_form", form)
    a = m.forward_tokens(toks, 0, list(range(n)))
    assert np.array_equal(a, m.forward_tokens(toks, 0, list(range(n))))
    m.set_option("tensor_cores", 0)
    b = m.forward_tokens(toks, 0, list(range(n)))
    assert G.rel_rms(a, b) < 5e-3
    m.close()
