"""Columns long enough that a block of a pass takes several tiles of one of them: the full histogram's table
and its lists of NaNs kept from tile to tile, the loops over an item's tiles of packing, both split passes and
the delta sums at every element width.  Blobs against the oracle byte for byte, decodes bit for bit, both
schedules (run_batch)."""
import numpy as np
import pytest

import oracle as OR
from test_batch_gpu import run_batch

pytestmark = pytest.mark.gpu

TILE = 4096  # the histogram tile of these tables
PATHS = [[OR.DICT, OR.NONE, OR.NONE], [OR.CONST, OR.NONE]]


def fallback(kind, n, npt):
    """columns whose most frequent values only the full histogram tells"""
    if kind == "equal":  # 5000 values of nearly one frequency: a table of one block holds them
        return (np.arange(n, dtype=np.int64) * 7919 % 5000 - 2500).astype(npt)
    if kind == "unique":  # no table holds them: flushed inside the column
        return (np.arange(n, dtype=np.int64) * 2654435761 % 2147483647 - 7).astype(npt)
    # all different, and NaNs of both signs; the four smallest in several tiles, three of them in those of one
    # block (of two per SM)
    x = (np.arange(n) + 0.5).astype(npt)
    bits = x.view(np.uint64 if x.itemsize == 8 else np.uint32)
    exp, man = (0x7ff << 52, 52) if x.itemsize == 8 else (0xff << 23, 23)
    sign = 1 << (8 * x.itemsize - 1)
    some = np.arange(100, n, 9973)
    bits[some] = np.array([(exp | (1 << man - 1) | (int(i) & 0xffff) | (sign if i & 1 else 0)) for i in some], bits.dtype)
    payload = (1 << man) - 1
    for k, tile in enumerate([5, 5 + 148, 5 + 2 * 148, 5 + 4 * 148]):
        bits[tile * TILE + 17 * k] = exp | sign | (payload - k)  # the largest magnitudes of the negative side
        bits[tile * TILE + 17 * k + 3] = exp | sign | (payload // 2 - k)
    return x


@pytest.mark.parametrize("dt", [OR.SHORT, OR.INT, OR.TIME, OR.FLOAT, OR.DOUBLE], ids=["short", "int", "time", "float", "double"])
def test_full_histogram_over_many_tiles(G, O, dt):
    npt = OR.NP_TYPES[dt]
    kinds = ["equal"] + (["unique"] if dt != OR.SHORT else []) + (["nans"] if dt in (OR.FLOAT, OR.DOUBLE) else [])
    cols, trees = [], []
    for kind in kinds:
        for path in PATHS:
            cols.append(fallback(kind, 3_000_001, npt))
            trees.append(G.tree_from_path(path, dt))
    b, _, _ = run_batch(G, O, cols, [dt] * len(cols), trees, steps=2,
                        tuning=G.tuning(hist_tile=TILE))  # several tiles for each resident block
    full = sum(by for name, _, by, _ in b.profile(True) if name == "hist_full")
    assert full == sum(x.nbytes for x in cols)  # no column was proven


@pytest.mark.parametrize("dt", [OR.CHAR, OR.SHORT, OR.TIME], ids=["char", "short", "time"])
def test_item_loops_of_other_widths(G, O, rng, dt):
    n = 6_400_013
    npt = OR.NP_TYPES[dt]
    x = rng.integers(0, 90, n).astype(npt)
    x[rng.integers(0, n, n // 20)] = 120
    walk = np.cumsum(rng.integers(-3, 4, n)).astype(npt)
    cases = [(x, [OR.PATCH, OR.AFL, OR.NONE, OR.NONE]), (x, [OR.AFL, OR.NONE]), (walk, [OR.DELTA, OR.NONE]),
             (x, [OR.DICT, OR.NONE, OR.NONE])]
    if dt != OR.CHAR:
        cases.append((walk, [OR.DELTA, OR.SCALE, OR.AFL, OR.NONE]))
    run_batch(G, O, [c for c, _ in cases], [dt] * len(cases), [G.tree_from_path(p, dt) for _, p in cases])


@pytest.mark.parametrize("dt", [OR.CHAR, OR.SHORT, OR.INT, OR.TIME, OR.DOUBLE], ids=["char", "short", "int", "time", "double"])
def test_few_values_of_one_frequency_need_no_full_histogram(G, O, rng, dt):
    """some hundred equally frequent values, and 1 % others: the candidates tell the most frequent ones"""
    npt = OR.NP_TYPES[dt]
    cols, trees = [], []
    for k, n in [(100, 20_011), (100, 400_003), (256, 400_003), (256, 1_000_001)]:
        x = rng.integers(0, k, n)
        if np.dtype(npt).itemsize >= 4:
            x[rng.integers(0, n, n // 100)] = rng.integers(0, 1 << 31, n // 100)
        cols.append((x % (100 if dt == OR.CHAR else 1 << 31)).astype(npt))
        trees.append(G.tree_from_path(PATHS[0], dt))
    b, _, _ = run_batch(G, O, cols, [dt] * len(cols), trees)
    assert sum(by for name, _, by, _ in b.profile(True) if name == "hist_full") == 0
