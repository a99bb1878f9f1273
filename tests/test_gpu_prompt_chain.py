"""Prompt portions with their kernels chained by programmatic dependent launch (option "prompt_pdl") and without: the same
logits to the bit, whole and in portions, for every folder architecture, in both number formats.  Only Genetar's are chained; for
the others the option has no effect, and this holds them to giving the same bits pass after pass."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arch", ["tudatar", "rupenex", "badepel", "bolapel", "lutesun"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_chained_or_not(gpu_lib, tmp_path, arch, dtype):
    T = importlib.import_module(f"test_gpu_{arch}")
    n = 600   # long enough for the tensor-core attention
    cfg = T.mixed_cfg()
    toks = T.tokens_for(cfg, n)
    W = T.O.random_weights(cfg, seed=1)
    m = gpu_lib.Transformer.open(T.O.write_model(str(tmp_path / "m"), cfg, W), dtype=dtype, max_tokens=n)
    want = [0, 1, 299, 300, n - 1]
    got = []
    for chained in (0, 1, 1):
        m.set_option("prompt_pdl", chained)
        whole = m.forward_tokens(toks, 0, want)
        parts = [m.forward_tokens(toks[a:b], a, [b - a - 1]) for a, b in ((0, 40), (40, 42), (42, 590), (590, n))]
        got.append(np.concatenate([whole] + parts))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_chained_or_not_genetar(gpu_lib, tmp_path, dtype):
    import genetar_oracle as G
    n = 700
    cfg = G.make_config([G.attention_layer(k, heads=8, kv_heads=2, dim=64, vdim=64, ff=640) for k in ("attention", "attention_2")], width=512, vocab=300)
    W = G.random_weights(cfg, seed=2)
    toks = np.random.default_rng(5).integers(0, 300, n).tolist()
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype=dtype, max_tokens=n)
    got = []
    for chained in (0, 1, 1):
        m.set_option("prompt_pdl", chained)
        got.append(np.concatenate([m.forward_tokens(toks, 0, [0, 350, n - 1])] + [m.forward_tokens(toks[a:b], a, [b - a - 1]) for a, b in ((0, 200), (200, 203), (203, n))]))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    m.close()
