"""The one-row product (gemv_rows_kernel) at the edges of its split: rows that are one 16-byte piece, rows whose pieces do not fill a
round of 32 lanes or a slice of K, one row more or less than a task, K split over two to eight warps, rows that do not start
on 16-byte boundaries, rows of one and two rounds (one and two pieces in flight).  Decode steps of one-layer Genetar models against the float64 implementation, held to the tolerances of
test_gpu_genetar.py (2e-4 and 4e-2 of the logits' root mean square)."""
import numpy as np
import pytest

import genetar_oracle as G

pytestmark = pytest.mark.gpu
TOL = {"float32": 2e-4, "bfloat16": 4e-2}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,ff,vocab", [(8, 8, 5), (72, 1, 3), (264, 136, 61), (1032, 520, 65), (520, 2056, 64), (512, 4104, 33), (27, 23, 10),
                                            (256, 512, 61), (128, 264, 33)])
def test_decode_steps(gpu_lib, tmp_path, dtype, width, ff, vocab):
    check_one_layer(gpu_lib, tmp_path, dtype, width, ff, vocab)


def check_one_layer(gpu_lib, tmp_path, dtype, width, ff, vocab):
    cfg = G.make_config([G.attention_layer("attention_2", heads=4, kv_heads=2, dim=16, vdim=16, ff=ff, v_mix=False)], width=width, vocab=vocab)
    W = G.random_weights(cfg, seed=width + ff)
    toks = np.random.default_rng(ff).integers(0, vocab, 6).tolist()
    want, _ = G.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(G.write_model(str(tmp_path / "m"), cfg, W), dtype=dtype, max_tokens=16)
    got = np.stack([m.forward(t, i).copy() for i, t in enumerate(toks)])
    assert G.rel_rms(got, want) < TOL[dtype]
    m.close()


@pytest.mark.parametrize("dtype,width", [("float32", 12288), ("bfloat16", 24448)])
def test_input_rows_of_about_48_kb(gpu_lib, tmp_path, dtype, width):
    """normalised rows whose shared memory reaches 48 KB only together with the kernel's own arrays"""
    check_one_layer(gpu_lib, tmp_path, dtype, width, 8, 5)


def test_widest_f32_input_rows(gpu_lib, tmp_path):
    """58048 columns leave room for the sums of a K split in an SM's 227 KB, 58052 do not"""
    for width in (58048, 58052):
        check_one_layer(gpu_lib, tmp_path, "float32", width, 8, 5)
