"""The tensor-core prompt attention (csrc/attn_tensor.cuh) where its tiles end: query rows and keys around whole tiles of 128 (and of the
16, 32 and 64 keys its steps take), head sizes that fill one or two operand boxes or only part of one, grouped heads that do not divide a
tile, prompts cut in portions.  One-layer Genetar models in float32 against the float64 implementation, held to that mode's 2e-4 of the
logits' root mean square (test_gpu_genetar.py); windows, chunks, penalties, sinks and gates through the mixed models of the other test
files, held to theirs.  These calls are too small to take the kernel by themselves: option "attn_tiles" 2."""
import importlib

import numpy as np
import pytest
import torch

import genetar_oracle as G
import rupenex_oracle as R
import tudatar_oracle as Tu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,n", [
    (4, 1, 64, 64, 32),     # exactly one tile of rows
    (4, 1, 64, 64, 33),     # one row more
    (1, 1, 64, 64, 257),    # key tiles: two whole ones and one key
    (3, 1, 128, 128, 65),   # 42 tokens x 3 heads in a tile of 128 rows; one key beyond a box of values
    (2, 2, 128, 64, 130),   # latent attention's shape
    (2, 2, 96, 96, 129),    # a box and a half
    (2, 1, 72, 72, 70),     # ends inside a step of 16
    (2, 1, 112, 20, 400),   # both groups of warps with several tiles
    (2, 1, 20, 4, 90),      # one piece of values
    (2, 1, 10, 6, 80),      # sizes that are not whole 16-byte pieces
    (20, 1, 32, 32, 9),     # more grouped heads than a tile takes at once
    (2, 2, 16, 128, 2),     # the fewest rows
])
def test_tile_edges(gpu_lib, tmp_path, heads, kv_heads, dim, vdim, n):
    cfg = G.make_config([G.attention_layer("attention_2", heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, ff=0, v_mix=False, scale=0.3, rot_dims=4)])
    W = G.random_weights(cfg, seed=dim + n, qk_gain=2.0)
    toks = np.random.default_rng(n).integers(0, cfg["vocab"], n).tolist()
    want, _ = G.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=400)
    m.set_option("attn_tiles", 2)
    whole = m.forward_tokens(toks, 0, list(range(n)))
    assert G.rel_rms(whole, want) < 2e-4
    cut = max(1, n // 2 - 3)   # a portion that starts inside a tile
    parts = np.concatenate([m.forward_tokens(toks[:cut], 0, list(range(cut))), m.forward_tokens(toks[cut:], cut, list(range(n - cut)))])
    assert G.rel_rms(parts, want) < 2e-4
    m.close()


@pytest.mark.parametrize("arch", ["tudatar", "rupenex", "badepel", "bolapel", "lutesun"])
def test_forms_of_the_other_models(gpu_lib, tmp_path, arch):
    """windows with and without kept keys, blocks, penalties, sinks, gates, expanded latent heads: a prompt over two key tiles whole,
    and in portions that start inside a tile"""
    T = importlib.import_module(f"test_gpu_{arch}")
    n = 150
    cfg = T.mixed_cfg()
    toks = T.tokens_for(cfg, n)
    W = T.weights_for(cfg, toks, seed=1) if hasattr(T, "weights_for") else T.O.random_weights(cfg, seed=1)
    want, _ = T.O.forward(cfg, W, toks)
    m = T.open_model(gpu_lib, tmp_path, cfg, W, "float32")
    m.set_option("attn_tiles", 2)
    assert T.O.rel_rms(m.forward_tokens(toks, 0, list(range(n))), want) < T.TOL["float32"]
    cuts = [0, 67, 74, 140, n]
    parts = [m.forward_tokens(toks[a:b], a, list(range(b - a))) for a, b in zip(cuts, cuts[1:])]
    assert T.O.rel_rms(np.concatenate(parts), want) < T.TOL["float32"]
    m.close()


def test_scores_as_low_as_the_other_kernels_take_them(gpu_lib, tmp_path):
    """a row whose only visible keys score between -1e30 and -1e30 / log2(e): still an average of their values"""
    cfg = G.make_config([G.attention_layer("attention", heads=4, kv_heads=4, dim=16, vdim=16, ff=0, v_mix=False, scale=-5e28, softcap=None)], bigram=None)
    W = G.random_weights(cfg, seed=3)
    W["l0.mix.k"] = W["l0.mix.q"]   # q . k of a token with itself is 16: its score is -8e29
    toks = np.random.default_rng(3).integers(0, cfg["vocab"], 40).tolist()
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=64)
    m.set_option("attn_tiles", 0)
    want = m.forward_tokens(toks, 0, list(range(40)))
    m.set_option("attn_tiles", 2)
    got = m.forward_tokens(toks, 0, list(range(40)))
    assert np.isfinite(want[0]).all() and np.isfinite(got).all()
    assert G.rel_rms(got[0], want[0]) < 2e-4
    m.close()


@pytest.mark.parametrize("keep_first", [0, 200])
def test_hidden_tiles_and_sinks_that_are_off(gpu_lib, tmp_path, keep_first):
    """a prompt longer than its window by several key tiles, which both groups of warps skip or walk (those of kept first keys included), in heads
    whose sink adds nothing (-inf, the lowest value of the weights' type) or something; whole, and in portions behind hidden tiles"""
    n = 900
    cfg = R.make_config([R.attention_layer(heads=8, kv_heads=2, dim=16, vdim=20, size=400, keep_first=keep_first, mlp=None)])
    W = R.random_weights(cfg, seed=6, gain=2.0)
    W["l0.mix.sink"] = np.array([-np.inf, -3.3895313892515355e38, 0.0, 2.0, -1e30, -np.inf, 5.0, -40.0])
    toks = np.random.default_rng(keep_first).integers(0, cfg["vocab"], n).tolist()
    want, _ = R.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(R.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=n)
    assert R.rel_rms(m.forward_tokens(toks, 0, list(range(n))), want) < 2e-4
    cuts = [0, 520, 580, 582, 850, n]
    parts = [m.forward_tokens(toks[a:b], a, list(range(b - a))) for a, b in zip(cuts, cuts[1:])]
    assert R.rel_rms(np.concatenate(parts), want) < 2e-4
    m.close()


@pytest.mark.parametrize("softcap", [None, 8.0])
@pytest.mark.parametrize("dim", [10, 72])
def test_a_key_that_scores_minus_infinity(gpu_lib, tmp_path, dim, softcap):
    """a token whose key is beyond f32 in one dimension and scores -inf for every row: no weight (or, capped, the least one), as in 64 bits"""
    n = 560   # long enough to take the kernel by itself
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=dim, vdim=dim, ff=0, v_mix=False, scale=0.3, softcap=softcap, rot_dims=4)], bigram=None)
    W = G.random_weights(cfg, seed=8, qk_gain=2.0)
    W["embed"][:, 0], W["embed"][:, 1], W["l0.norm1"][0] = 1.0, 0.0, 1.0
    W["embed"][60, 1] = -8.0
    for name, column, value in (("q", 0, 1.0), ("k", 1, 2.0 ** 127)):
        for h in range(4 if name == "q" else 2):
            row = W["l0.mix." + name][h * dim + 7]
            row[:] = 0.0
            row[column] = value
    toks = np.random.default_rng(n).integers(0, 60, n)
    toks[[5, 130, 131, 300, 558]] = 60
    toks = toks.tolist()
    want, _ = G.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=n)
    assert G.rel_rms(m.forward_tokens(toks, 0, list(range(n))), want) < 2e-4
    parts = [m.forward_tokens(toks[a:b], a, list(range(b - a))) for a, b in ((0, 531), (531, n))]
    assert G.rel_rms(np.concatenate(parts), want) < 2e-4
    m.close()


def test_rows_do_not_see_later_tokens_that_are_no_numbers(gpu_lib, tmp_path):
    """a NaN among the keys and values of a later token of the same tile: the rows before it are what they are without it"""
    n, at = 700, 600
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=24, vdim=40, ff=0, v_mix=False, scale=0.3, rot_dims=4)], bigram=None)
    W = G.random_weights(cfg, seed=9, qk_gain=2.0)
    W["embed"][60, 3] = np.nan
    toks = np.random.default_rng(n).integers(0, 60, n).tolist()
    want, _ = G.forward(cfg, W, toks[:at])
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=n)
    toks[at] = 60
    got = m.forward_tokens(toks, 0, list(range(n)))
    assert G.rel_rms(got[:at], want) < 2e-4
    assert np.isnan(got[at:]).all()
    m.close()


@pytest.mark.parametrize("form", ["kept keys and sinks", "kept keys up to the window", "penalty"])
def test_windowed_rows_before_a_token_that_is_no_number(gpu_lib, tmp_path, form):
    """the same for rows with a window, kept first keys, sinks that are on and off, a distance penalty: rows 256 .. 286 are computed again, over the keys they see"""
    n, at = 320, 287
    if form == "penalty":
        O = Tu
        cfg = Tu.make_config([Tu.window_layer(heads=8, kv_heads=2, dim=12, vdim=20, window=90, mlp=None)])
    else:
        O = R
        cfg = R.make_config([R.attention_layer(heads=8, kv_heads=2, dim=12, vdim=20, size=90, keep_first=20 if form.endswith("sinks") else 250, mlp=None)])
    W = O.random_weights(cfg, seed=6, gain=2.0)
    if O is R:
        W["l0.mix.sink"] = np.array([-np.inf, -3.3895313892515355e38, 0.0, 2.0, -1e30, -np.inf, 5.0, -40.0])
    toks = np.random.default_rng(3).integers(0, 60, n).tolist()
    want, _ = O.forward(cfg, W, toks[:at])
    W["embed"][60] = np.nan
    toks[at] = 60
    m = gpu_lib.Transformer.open(O.write_model(str(tmp_path / "m"), cfg, W), dtype="float32", max_tokens=n)
    m.set_option("attn_tiles", 2)
    got = m.forward_tokens(toks, 0, list(range(n)))
    assert O.rel_rms(got[:at], want) < 2e-4
    assert O.rel_rms(got[256:at], want[256:]) < 2e-4
    assert np.isnan(got[at:]).all()
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_first_prompt_finds_the_room_for_its_pieces(gpu_lib, tmp_path, dtype):
    """the pieces of keys, values and (float32) rows are given room when the model is loaded: where everything else is allocated already, the first
    prompt that takes the tensor-core kernels leaves the free memory as it is"""
    n = 600
    cfg = G.make_config([G.attention_layer("attention_2", heads=8, kv_heads=8, dim=64, vdim=64, ff=4096)], width=1024, vocab=64)
    folder = G.write_model(str(tmp_path / "m"), cfg, G.random_weights(cfg, seed=1))
    toks = np.random.default_rng(1).integers(0, 64, n).tolist()
    loads_the_kernels = gpu_lib.Transformer.open(folder, dtype=dtype, max_tokens=n)
    loads_the_kernels.forward_tokens(toks, 0, [n - 1])
    m = gpu_lib.Transformer.open(folder, dtype=dtype, max_tokens=n)
    for name, value in (("attn_tiles", 1), ("gemm_split", 0)):
        m.set_option(name, value)
    m.forward_tokens(toks, 0, [n - 1])
    before = torch.cuda.mem_get_info()[0]
    for name in ("attn_tiles", "gemm_split"):
        m.set_option(name, -1)
    assert np.array_equal(m.forward_tokens(toks, 0, [n - 1]), loads_the_kernels.forward_tokens(toks, 0, [n - 1]))
    assert torch.cuda.mem_get_info()[0] == before
    m.close()
    loads_the_kernels.close()
