"""A chained prompt (programmatic dependent launches) has at most two kernels in flight: every kernel that one can hold lets its successor start only behind its
own wait.  What would go wrong otherwise is not to be provoked on a GPU, so this reads the kernels."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lm.rs_b200", "csrc")
# every kernel of a Genetar prompt but its first, the embedding, which is an ordinary launch, and the one-row product of a head of one row, its last
KERNELS = {"dense_ops.cuh": ["rmsnorm_rows_kernel", "gemm_tiled_kernel", "qkv_post_kernel", "attn_rows_kernel"], "attn_tiles.cuh": ["attn_tile_kernel"],
           "attn_tensor.cuh": ["attn_split_kernel", "attn_tensor_kernel"], "dense_gemm_f32.cuh": ["gemm_f32_kernel"],
           "dense_gemm_split.cuh": ["split_rows_kernel", "gemm_split_kernel"], "dense_gemm.cuh": ["gemm_bf16_tc_kernel", "gemm_bf16_pair_kernel"]}


@pytest.mark.parametrize("file,kernel", [(f, k) for f, ks in KERNELS.items() for k in ks])
def test_waits_before_it_launches(file, kernel):
    text = open(os.path.join(CSRC, file)).read()
    start = re.search(rf"__launch_bounds__\([^\n]*\)\s+{kernel}\(", text).start()
    calls = re.findall(r"pdl_(wait|launch|enter)\(([^;]*)\);", text[start:text.index("\n}\n", start)])
    names = [c[0] for c in calls]
    assert names in (["wait", "launch"], ["wait", "wait", "launch"], ["enter"])   # (a grouped product also waits for its row ranges)
    if names == ["enter"]:   # launches first in steps of one token only
        assert calls[0][1] in ("gridDim.x == 1", "p.T == 1")
