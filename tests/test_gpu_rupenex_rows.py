"""Rows of Rupenex prompts at the edges of their kernels: group norms with parts a warp holds (up to 512 columns) and longer ones, convolutions of four taps
(a sliding window) and of other widths over runs that end inside a block of four tokens, layer norms of rows a CTA holds in registers (up to 4096
columns) and longer, and more chosen experts than are loaded at a time.  Against the float64 implementation, with the tolerances of test_gpu_rupenex.py;
in bfloat16 the routers choose all of their outputs, as there."""
import numpy as np
import pytest

import rupenex_oracle as O
from test_gpu_rupenex import TOL

pytestmark = pytest.mark.gpu
# heads, vdim, norm groups (part = heads * vdim / groups), taps, width, tokens
CASES = [(8, 64, 1, 4, 40, 17), (8, 65, 1, 4, 40, 5), (8, 66, 2, 4, 260, 33), (4, 10, 2, 3, 41, 18), (4, 10, 4, 5, 256, 2), (4, 8, 1, 4, 4096, 3), (4, 8, 1, 2, 4100, 3)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,vdim,groups,taps,width,n", CASES)
def test_rows_at_the_edges(gpu_lib, tmp_path, heads, vdim, groups, taps, width, n, dtype):
    moe = O.moe(experts=6, identity=2, top=5 if dtype == "float32" else 8, ff=24, shared=24)
    cfg = O.make_config([O.ssm_layer(heads=heads, vdim=vdim, state=12, groups=2, conv=taps, norm_groups=groups, mlp=moe)], width=width, vocab=50)
    toks = np.random.default_rng(9).integers(0, 50, n).tolist()
    for seed in range(3, 23):   # weights without a near-tie between experts
        W = O.random_weights(cfg, seed=seed)
        if dtype == "bfloat16" or O.clear_choices(cfg, W, toks, 1e-4):
            break
    else:
        pytest.fail("no seed without a near-tie between experts")
    want, _ = O.forward(cfg, W, toks)
    m = gpu_lib.Transformer.open(O.write_model(str(tmp_path / "m"), cfg, W), dtype=dtype, max_tokens=64)
    for warps in (0, 1):   # (prompts as short as these take a CTA per part; parts over 512 columns always do)
        m.set_option("group_norm_warps", warps)
        assert O.rel_rms(m.forward_tokens(toks, 0, list(range(n))), want) < TOL[dtype]
    if n > 2:   # in two portions: the convolution continues from its tail
        cut = n // 2
        parts = np.concatenate([m.forward_tokens(toks[:cut], 0, list(range(cut))), m.forward_tokens(toks[cut:], cut, list(range(n - cut)))])
        assert O.rel_rms(parts, want) < TOL[dtype]
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("at", [5, 6, 7, 8, 16])
def test_a_token_without_numbers_spoils_no_earlier_row(gpu_lib, tmp_path, dtype, value, at):
    """loads run ahead of the rows they belong to (four tokens in the convolution, four experts in the sums)"""
    cfg = O.make_config([O.ssm_layer(heads=8, vdim=64, state=12, groups=2, norm_groups=1, mlp=O.moe(experts=4, identity=1, top=5, ff=24, shared=24))], width=40, vocab=50)
    W = O.random_weights(cfg, seed=3)
    toks = np.random.default_rng(2).integers(0, 49, 19).tolist()
    m = gpu_lib.Transformer.open(O.write_model(str(tmp_path / "a"), cfg, W), dtype=dtype, max_tokens=64)
    clean = m.forward_tokens(toks, 0, list(range(19)))
    m.close()
    W["embed"][49, 7] = value
    toks[at] = 49
    m = gpu_lib.Transformer.open(O.write_model(str(tmp_path / "b"), cfg, W), dtype=dtype, max_tokens=64)
    for warps in (0, 1):
        m.set_option("group_norm_warps", warps)
        got = m.forward_tokens(toks, 0, list(range(19)))
        assert np.array_equal(got[:at], clean[:at]) and np.isnan(got[at]).all()
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,vdim,groups,n", [(8, 64, 1, 17), (8, 64, 2, 2), (3, 171, 1, 9), (8, 65, 1, 5), (4, 10, 4, 33), (5, 1, 5, 3)])
def test_group_norm_sums_in_one_order(gpu_lib, tmp_path, dtype, heads, vdim, groups, n):
    """a warp per part or a CTA per part: the same bits"""
    cfg = O.make_config([O.ssm_layer(heads=heads, vdim=vdim, state=8, groups=1, norm_groups=groups, mlp=None)], width=40, vocab=50)
    toks = np.random.default_rng(4).integers(0, 50, n).tolist()
    m = gpu_lib.Transformer.open(O.write_model(str(tmp_path / "m"), cfg, O.random_weights(cfg, seed=6)), dtype=dtype, max_tokens=64)
    got = []
    for warps in (1, 0):
        m.set_option("group_norm_warps", warps)
        got.append(m.forward_tokens(toks, 0, list(range(n))))
    assert np.array_equal(*got)
    m.close()
