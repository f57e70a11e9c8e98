"""Few tokens of a SwitchGLU by pairs or by expert (csrc/exl3_moe_plan.h), compiled for the host: the tiles of the slowest CTA
against the tables' layout, and calls on both sides of the line with what they took."""

from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    out = tmp_path_factory.mktemp("emul") / "libmoe_plan_emul.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(HERE / "host_emul" / "moe_plan_emul.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.emul_by_expert.argtypes = [ctypes.c_int64] * 4 + [ctypes.c_int]
    lib.emul_most_tiles.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int]
    return lib


def test_tiles_of_the_slowest_cta(emul):
    """Tables as moe_prefill_tables_kernel writes them, a gate and an up table one after the other, two column halves an entry;
    CTA c of the tile kernel takes items c, c + 147, ..."""
    for hit, slots, cols, sets in ((1, 1, 128, 1), (50, 64, 384, 2), (68, 128, 384, 2), (68, 128, 1664, 1), (101, 256, 512, 2), (8, 8, 2048, 1)):
        per_slot = (cols + 255) // 256
        items = [t for t in range(sets * slots * per_slot * 2)
                 if t // 2 // per_slot % slots < hit and 256 * (t // 2 % per_slot) + 128 * (t % 2) < cols]
        count = [0] * 147
        for t in items:
            count[t % 147] += 1
        assert emul.emul_most_tiles(hit, slots, cols, sets) == max(count)


@pytest.mark.parametrize("tokens,experts,d,h,k,by_expert", [
    # us by pairs / by expert
    (16, 256, 2048, 512, 4, True),        # 132 / 118
    (16, 64, 2048, 512, 4, True),         # 131 / 82
    (16, 64, 1024, 256, 4, True),         # 44 / 41
    (12, 256, 2048, 512, 4, False),       # 105 / 107
    (12, 128, 1664, 384, 4, False),       # 68 / 75
    (14, 128, 1408, 384, 2, False),       # 70 / 83
    (12, 64, 1408, 384, 3, False),        # 58 / 62
    (6, 64, 2048, 512, 2, False),         # 58 / 67
    (1, 256, 2048, 512, 4, False),
    (16, 1025, 2048, 512, 4, False),      # no tables by expert
    (1, 1, 2048, 512, 4, False),
    (16, 1, 2048, 512, 4, True),
])
def test_line_between_the_two_ways(emul, tokens, experts, d, h, k, by_expert):
    assert emul.emul_by_expert(8 * tokens, experts, d, h, k) == by_expert


def test_the_gpu_test_lies_on_both_sides(emul):
    from test_gpu_fused_moe import FEW_TOKENS

    for k, tokens, e, d, h, kk, by_expert in FEW_TOKENS:
        assert emul.emul_by_expert(tokens * kk, e, d, h, k) == by_expert, (k, tokens)
    assert not emul.emul_by_expert(2**20 + 1, 64, 2048, 512, 4)
