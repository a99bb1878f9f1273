"""A wait of the tensor-core kernels on a barrier where nothing arrives ends within seconds, and the status word says which kernel and barrier it was.  The kernels'
own barriers cannot be made to miss an arrival, so the wait itself is compiled into a program of its own (one thread, one barrier)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_wait_that_runs_out(tmp_path):
    exe = str(tmp_path / "bounded_wait")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I", os.path.join(os.path.dirname(HERE), "lm.rs_b200", "csrc"),
                           "-o", exe, os.path.join(HERE, "bounded_wait.cu")])
    rows = [line.split("|") for line in subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines()]
    assert [r[0] for r in rows] == ["0", "1", "0"]
    ms = [int(r[1]) for r in rows]
    assert 2000 <= ms[0] < 10000 and ms[1] < 100 and ms[2] < 1000
    assert rows[0][2] == "attn_tensor_kernel gave up waiting for scores (device status 778)"
    assert rows[1][2] == "" and rows[2][2] == "gemm_bf16_pair_kernel gave up waiting for the sums (device status 515)"   # the first to give up is named
