"""The launch plan of the dense GEMM (csrc/exl3_gemm_plan.h), compiled for the host: the slowest CTA counted
without walking its segments, the choice among token and CTA counts, and what a plan costs on the host."""

from __future__ import annotations

import ctypes
import random
import subprocess
import time
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
TOKENS = [(256, 384), (240, 368), (224, 368), (208, 352), (192, 336)]      # tokens of an ordinary and a wide tile, K = 4 .. 8

ROOM = 162 * 1024                   # shared memory of the rings; a stage of packed tiles is K KiB


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    out = tmp_path_factory.mktemp("emul") / "libgemm_plan_emul.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out),
                    str(HERE / "host_emul" / "gemm_plan_emul.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    i, l = ctypes.c_int, ctypes.c_int64
    for f in (lib.emul_plan, lib.exhaustive_plan):
        f.argtypes = [l, l, i, i, i, i, i, ctypes.c_void_p]
        f.restype = None
    lib.emul_countable.argtypes = [l, l, i, i, i, i, i]
    lib.emul_slowest.argtypes, lib.emul_slowest.restype = [l, i, i, i], l
    return lib


def _plan(f, *args):
    out = (ctypes.c_int * 5)()
    f(*args, out)
    return tuple(out)


def test_slowest_cta_equals_the_walk_over_its_segments(emul):
    rng = random.Random(1)
    for _ in range(4000):
        nks = rng.choice([1, 2, 3, 8, 46, 80, 272, rng.randint(1, 300)])
        units = nks * rng.randint(1, 2000)
        g = rng.randint(1, min(148, units))
        assert emul.emul_slowest(units, nks, g, 0) == emul.emul_slowest(units, nks, g, 1), (units, nks, g)


def test_choice_equals_the_exhaustive_search(emul):
    rng = random.Random(2)
    for n in range(1500):
        rows = round(2 ** rng.uniform(3, 14 if n % 10 else 17))
        tiles_n, nks = rng.randint(1, 272), 2 * rng.randint(1, 136)
        tok, wide = rng.choice(TOKENS)
        room = rng.choice([0, tok, 384, 384, 384])
        if rows * tiles_n > 4_000_000:
            continue
        args = (rows, tiles_n, nks, rng.choice([148, 148, 148, 132, 20]), tok, wide, room)
        assert _plan(emul.emul_plan, *args) == _plan(emul.exhaustive_plan, *args), args


def test_every_shape_that_fits_a_gpu_can_be_counted(emul):
    """rows x in x out beyond 2^31 k-steps of tiles: 42,000 rows of 400,000 x 400,000 (K = 1: 120 GB in all) and the
    like are dealt in whole tiles, which are counted; k-steps of shared tiles stay within 32 bits."""
    for rows, inf, outf in ((42_000, 400_000, 400_000), (65_536, 262_144, 262_144), (20_000, 800_000, 500_000), (8_000_000, 4096, 4096),
                            (1, 16_777_216, 65_536), (1, 65_536, 16_777_216), (500, 2_000_000, 500_000)):
        for tok, wide in TOKENS:
            args = (rows, outf // 128, inf // 64, 148, tok, wide, 384)
            assert emul.emul_countable(*args), args
            tok_, tiles_m, grid, split, _ = _plan(emul.emul_plan, *args)
            assert tiles_m * tok_ >= rows and (not split or tiles_m * (outf // 128) * (inf // 64) < 2**31)


def test_the_gpu_tests_reach_every_form_of_the_kernel(emul):
    from test_gpu_gemm import FORMS

    for rows, inf, outf, k, cb, form in FORMS:
        _, tiles_m, grid, _, is_wide = _plan(emul.emul_plan, rows, outf // 128, inf // 64, 148, *TOKENS[max(0, k - 4)], 384)
        assert form == ("wide" if is_wide else "ahead" if tiles_m * (outf // 128) >= 2 * grid else "plain"), (rows, inf, outf, k)


def test_a_plan_costs_less_than_a_launch(emul):
    """A new row count is planned anew; an exhaustive search of these takes milliseconds each."""
    shapes = [(40, 80), (136, 80), (40, 272), (32, 64), (11, 46)]
    out = (ctypes.c_int * 5)()
    t0 = time.perf_counter()
    n = 0
    for rows in list(range(9, 400, 13)) + list(range(401, 8192, 401)):
        for tiles_n, nks in shapes:
            emul.emul_plan(rows, tiles_n, nks, 148, 256, 384, 384, out)
            n += 1
    assert (time.perf_counter() - t0) / n < 200e-6


def test_clusters_of_a_tile(emul):
    """Where the CTAs of a tile become a cluster: up to eight of them with at least four k-steps each, all on the chip at a time, no
    tile of more than 128 tokens, and never more CTAs than asked for."""
    emul.emul_joint.argtypes = [ctypes.c_int64, ctypes.c_int64] + [ctypes.c_int] * 6
    rng = random.Random(7)
    taken = set()
    for _ in range(3000):
        rows, tiles_n, nks = rng.randint(9, 400), rng.randint(1, 160), 2 * rng.randint(1, 136)
        most = rng.randint(1, 8)
        args = (rows, tiles_n, nks, 148, 256, 384, rng.choice([0, 384]))
        tok, tiles_m, _, split, _ = _plan(emul.emul_plan, *args)
        n = emul.emul_joint(*args, most)
        taken.add(n)
        assert n == 0 or (2 <= n <= most and 4 * n <= nks and split and tok <= 128 and tiles_m * tiles_n * n <= 148), (args, n)
    assert taken == {0, 2, 3, 4, 5, 6, 7, 8}
    assert emul.emul_joint(77, 40, 80, 148, 256, 384, 384, 8) == 3      # 5120 x 5120: three CTAs of 27 k-steps
    assert emul.emul_joint(77, 136, 80, 148, 256, 384, 384, 8) == 0     # 5120 x 17408: a CTA per tile


@pytest.mark.parametrize("k", range(1, 9))
def test_clusters_leave_room_for_the_rings(emul, k):
    """The sums that a cluster's CTAs exchange take shared memory from the rings: 96 of 162 KiB for seven CTAs and 128 tokens.
    Whatever the shape and however many clusters the device holds, two stages of activations fit beside eight of packed tiles."""
    seen = (ctypes.c_int * 9)()
    least = emul.emul_joint_stages(140, 148, *TOKENS[max(0, k - 4)], ROOM, 1024 * k, seen)
    assert least >= 2, list(seen)
    assert all(seen[n] for n in range(2, 9)), list(seen)


def test_the_gpu_tests_reach_clusters_of_each_size(emul):
    """By the number of k-steps, so that a device that holds fewer clusters of the largest sizes does not change them."""
    from test_gpu_gemm import CLUSTERS

    emul.emul_joint_beside.argtypes = [ctypes.c_int64, ctypes.c_int64] + [ctypes.c_int] * 8
    for inf, outf, k, cb, rows, n in CLUSTERS:
        assert emul.emul_joint_beside(rows, outf // 128, inf // 64, 148, *TOKENS[max(0, k - 4)], 384, ROOM, 1024 * k, 8) == n, (inf, outf, k, rows)
