"""The size rules of csrc/dense_dispatch.h at sizes where both sides were timed on a B200 (148 SMs): the rule may not take a kernel that
was more than 3 % slower than the other one.  Times in us per call and layer."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lm.rs_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    """runs C++ statements over the header and returns the integers they print"""
    folder = tmp_path_factory.mktemp("rules")

    def run(statements):
        src, exe = folder / "r.cpp", folder / "r"
        src.write_text('#include <cstdio>\n#include "dense_dispatch.h"\nusing namespace lmrs::dense;\nint main() {\n' + "\n".join(statements) + "\n}\n")
        subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
        return [int(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]
    return run


# heads, KV heads, head size, tokens, position: 16-row tiles, 64-row tiles
ATTENTION = [
    (32, 8, 64, 16, 2000, 262, 295),
    (32, 8, 64, 64, 500, 155, 166),
    (32, 8, 64, 128, 0, 120, 120),
    (32, 8, 64, 192, 2000, 345, 302),
    (32, 8, 64, 256, 0, 132, 121),
    (24, 8, 128, 32, 2000, 387, 492),
    (24, 8, 128, 64, 64, 154, 166),
    (24, 8, 128, 128, 1000, 307, 335),
    (24, 8, 128, 192, 500, 289, 245),
    (24, 8, 128, 256, 0, 181, 165),
    (32, 32, 96, 64, 2000, 373, 468),
    (32, 32, 96, 128, 500, 228, 240),
    (32, 32, 96, 192, 1000, 333, 325),
    (32, 32, 96, 256, 64, 210, 190),
    (16, 4, 64, 16, 1000, 159, 176),
    (16, 4, 64, 128, 2000, 244, 281),
    (16, 4, 64, 384, 2000, 342, 305),
    (16, 4, 64, 512, 0, 137, 133),
    (16, 16, 128, 64, 500, 188, 222),
    (16, 16, 128, 256, 1000, 303, 333),
    (16, 16, 128, 384, 0, 197, 186),
    (4, 2, 64, 64, 500, 114, 124),
    (4, 2, 64, 512, 0, 108, 116),
    (4, 2, 64, 768, 2000, 316, 324),
]


def test_attention_tiles(rules):
    calls = []
    for heads, kv, dim, T, pos, _, _ in ATTENTION:
        hc = min(heads // kv, 16)
        columns = kv * -(-heads // kv // hc)
        calls.append(f'printf("%d ", attn_large_tiles(148, {T}, {columns}, {hc}));')
    for row, large in zip(ATTENTION, rules(calls)):
        times = row[5:]
        assert times[large] <= 1.03 * min(times), row


def test_order_of_the_large_tiles(rules):
    """turns only where two CTAs share an SM: 114,688 bytes (128-wide heads) twice, 147,456 (192-wide keys, 128-wide values) once"""
    assert rules([f'printf("%d ", attn_order_turns_at(148, {b}));' for b in (114688, 115712, 115713, 147456)]) == [148, 148, 0, 0]


def test_ring_of_the_two_sm_products(rules):
    """clusters of four: 33 at once with one CTA per SM; more of them share SMs instead of forming a second wave"""
    assert rules([f'printf("%d ", gemm_whole_sm({n}, 33));' for n in (32, 33, 34, 37, 74)]) == [1, 1, 0, 0, 0]
