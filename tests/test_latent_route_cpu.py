"""Which kernel latent attention takes: the rule against what both took on a B200."""
import ctypes
import random

import numpy as np
import pytest

from conftest import pkg


@pytest.fixture(scope="module")
def lib():
    lib, i32 = pkg("_abi").lib(), ctypes.c_int32
    lib.b200_debug_latent_route.argtypes = [i32] * 6 + [ctypes.c_int64, i32]
    lib.b200_debug_latent_by_rows.argtypes = [i32] * 9
    return lib


ROWS, EITHER, RUNS = 0, 1, 2

# layout (own: rows of sequences of their own, one: rows of one sequence, long: one of that many tokens among rows of 600), row width and rank, heads, rows,
# tokens, splits that such a step asks for; us over runs with those splits, without splits, and by themselves
MEASURED = [
    ("own", 576, 512, 16, 1, 3000, 16, 54, 87, 25), ("own", 576, 512, 16, 8, 16000, 16, 126, 425, 70), ("one", 576, 512, 16, 8, 16000, 16, 95, 398, 62),
    ("own", 576, 512, 16, 16, 60000, 16, 482, 1537, 371), ("one", 576, 512, 16, 16, 16000, 16, 97, 384, 107), ("own", 576, 512, 16, 33, 3000, 9, 122, 97, 43),
    ("own", 576, 512, 16, 33, 64000, 9, 943, 1611, 422), ("one", 576, 512, 16, 33, 16000, 9, 106, 392, 109), ("own", 576, 512, 16, 74, 16000, 4, 479, 424, 238),
    ("one", 576, 512, 16, 74, 16000, 4, 151, 382, 201), ("own", 576, 512, 16, 100, 3000, 3, 208, 179, 96), ("one", 576, 512, 16, 100, 3000, 3, 87, 93, 86),
    ("one", 576, 512, 16, 100, 8000, 3, 124, 210, 201), ("own", 576, 512, 16, 100, 16000, 3, 732, 827, 403), ("one", 576, 512, 16, 100, 16000, 3, 183, 392, 385),
    ("own", 576, 512, 16, 148, 16000, 1, 840, 840, 440), ("one", 576, 512, 16, 148, 16000, 1, 386, 386, 387), ("own", 576, 512, 32, 18, 60000, 9, 564, 1473, 711),
    ("one", 576, 512, 32, 18, 16000, 9, 108, 383, 200), ("own", 576, 512, 64, 8, 60000, 10, 378, 1514, 365), ("one", 576, 512, 64, 18, 16000, 5, 136, 388, 201),
    ("own", 576, 512, 128, 4, 60000, 10, 210, 1451, 362), ("one", 576, 512, 128, 8, 16000, 5, 136, 386, 201), ("own", 576, 512, 128, 18, 60000, 3, 1023, 1508, 1398),
    ("one", 576, 512, 128, 18, 8000, 3, 126, 210, 201), ("long", 576, 512, 16, 33, 32000, 9, 167, 792, 202), ("long", 576, 512, 16, 64, 32000, 5, 253, 798, 387),
    ("long", 576, 512, 16, 100, 32000, 3, 368, 820, 756), ("long", 576, 512, 16, 148, 32000, 1, 818, 818, 758),
    ("own", 288, 256, 4, 148, 12000, 8, 318, 233, 207), ("one", 288, 256, 4, 148, 12000, 8, 69, 224, 172), ("one", 288, 256, 16, 74, 12000, 4, 93, 224, 94),
    ("own", 288, 256, 128, 18, 12000, 3, 112, 202, 182), ("own", 192, 128, 4, 148, 12000, 8, 276, 224, 131), ("one", 192, 128, 4, 148, 12000, 8, 55, 218, 119),
    ("own", 192, 128, 16, 74, 12000, 4, 141, 224, 80), ("own", 192, 128, 128, 18, 12000, 3, 87, 171, 119), ("one", 80, 64, 4, 148, 12000, 8, 50, 228, 98),
    ("own", 80, 64, 16, 33, 12000, 9, 99, 226, 35), ("own", 512, 512, 16, 74, 12000, 4, 335, 278, 166), ("own", 512, 512, 128, 18, 12000, 3, 251, 272, 273),
    ("own", 576, 512, 16, 512, 2000, 1, 433, 433, 256), ("own", 576, 512, 32, 512, 2000, 1, 432, 432, 404), ("own", 576, 512, 64, 160, 2000, 1, 202, 202, 284),
    ("own", 576, 512, 128, 512, 2000, 1, 931, 931, 1543), ("own", 192, 128, 128, 64, 3000, 1, 104, 104, 133)]


@pytest.mark.parametrize("layout,krow,rank,heads,T,ctx,splits,runs_split,runs_whole,rows", MEASURED)
def test_the_route_is_not_much_slower_than_the_other(lib, layout, krow, rank, heads, T, ctx, splits, runs_split, runs_whole, rows):
    route = lib.b200_debug_latent_route(T, heads, krow, rank, 128, splits, ctx + T, int(T * -(-heads // 16) > 148))
    tiles = {"own": T * -(-ctx // 64), "one": -(-T // 16) * -(-ctx // 64), "long": (T - 1) * 10 + -(-ctx // 64)}[layout]
    n_runs = -(-T // 16) if layout == "one" else T
    over = route == RUNS or (route == EITHER and not lib.b200_debug_latent_by_rows(T, heads, krow, rank, splits, 0, n_runs, ctx, tiles))
    took = runs_split if over else rows
    assert took <= 1.13 * min(rows, runs_split), (route, over)


def test_routes_of_forms(lib):
    r = lambda T=64, heads=16, krow=576, rank=512, bs=128, splits=1, longest=4096, own=0: lib.b200_debug_latent_route(T, heads, krow, rank, bs, splits, longest, own)   # noqa: E731
    assert r() == ROWS and r(T=148) == ROWS and r(T=149) == RUNS and r(T=149, own=1) == ROWS and r(T=4096, own=1) == ROWS
    assert r(heads=17, T=74) == ROWS and r(heads=17, T=75) == RUNS and r(heads=48, T=60, own=1) == RUNS and r(heads=48, T=49) == ROWS
    assert r(heads=130, T=40, own=1) == ROWS                                   # more heads than the kernel over runs takes
    assert r(bs=96) == RUNS and r(krow=577) == RUNS and r(rank=520, krow=584) == RUNS   # not this kernel's shapes
    assert r(T=100, splits=3, longest=3200) == ROWS and r(T=100, splits=3, longest=16384) == EITHER and r(T=100, splits=1, longest=1 << 20) == ROWS
    assert r(T=7, splits=16, longest=1 << 20) == ROWS                          # with splits of its own
    assert r(T=8, splits=16, longest=30000) == ROWS and r(T=8, splits=16, longest=1 << 20) == EITHER
    # rows of few heads and narrow ones as any others; a call with hardly any queries keeps its two launches
    assert r(T=64, heads=4, krow=80, rank=64) == ROWS and r(T=148, heads=1, krow=32, rank=16) == ROWS and r(T=1, heads=2) == ROWS
    assert r(T=2, heads=4, krow=80, rank=64) == RUNS and r(T=1, heads=1) == RUNS and r(T=3, heads=1, krow=80, rank=64) == ROWS
    # a window bounds what a row sees, whatever its context
    assert lib.b200_debug_latent_by_rows(100, 16, 576, 512, 3, 1024, 100, 32000, 100 * 500) == 1


def test_nothing_overflows(lib):
    for T, longest in ((1, 1 << 30), (148, 1 << 30), (148, 1 << 60), (1 << 16, 1 << 20)):
        assert lib.b200_debug_latent_route(T, 16, 576, 512, 128, 16, longest, 1) in (ROWS, EITHER, RUNS)
        assert lib.b200_debug_latent_by_rows(T, 16, 576, 512, 16, 0, T, min(longest, (1 << 31) - 1), (1 << 31) - 1) in (0, 1)


def test_the_devices_answer_is_rounded_step_by_step(lib):
    """Several kernels answer the same question apart: the rule over a grid of plans is what fp32 products and sums give, rounded one by one."""
    rng, f = random.Random(1), np.float32
    for _ in range(2000):
        T, heads, krow, splits = rng.randint(1, 148), rng.choice([1, 4, 16, 17, 40, 128]), rng.choice([80, 192, 288, 512, 576]), rng.randint(2, 16)
        rank, window, n_runs = min(krow, 512), rng.choice([0, 0, 512, 4096]), rng.randint(1, T)
        longest = rng.randint(1, 1 << rng.randint(1, 20))
        tiles = rng.randint(-(-longest // 64), n_runs * -(-longest // 64))
        groups, per = -(-heads // 16), min(128 // heads, 16)
        cluster = next(c for n, c in ((15, 8), (33, 4), (74, 2), (1 << 30, 1)) if T * groups <= n)
        by_row, by_run = f(4.2) + f(0.035) * f(krow), f(1.15) * max(f(16.5), f(0.043) * f(krow))
        row_key, row_tile = by_row / f(cluster), by_row * f(64) * f(groups) / f(148)
        fixed, run_key, run_item = f(10000) + f(54) * f(krow), by_run / f(splits), by_run * f(64) / f(splits)
        seen = window or (1 << 31) - 1
        most, walked = f(min(longest, seen)), min(f(tiles), f(seen // 64 + 2) * f(n_runs))
        parts, halves = -(-T // (n_runs * per)), 2 if rank > 256 else 1
        rounds = -(-(n_runs * parts * halves * splits) // 148)
        by_rows = max(row_key * most, row_tile * walked)
        run = max(run_key * most * f(n_runs), run_item * (walked * f(rounds)))
        want = by_rows * f(n_runs) <= fixed * f(n_runs) + run
        assert lib.b200_debug_latent_by_rows(T, heads, krow, rank, splits, window, n_runs, longest, tiles) == int(want)
