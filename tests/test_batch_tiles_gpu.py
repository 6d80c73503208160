"""The batched passes at the edges of their units and tiles: every column's blob equals the oracle's
byte for byte and decodes bit for bit (both batch schedules, run_batch).  Sizes lie around the 32-value
rows, the 1024-value warp units, the 8192- and 4096-value tiles and the 131072-value counting tiles."""
import numpy as np
import pytest

import oracle as OR
from test_batch_gpu import run_batch

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 1023, 1024, 1025, 4095, 4097, 8191, 8192, 8193, 16400, 32769, 131071, 131073, 262177]
IDS = {OR.CHAR: "char", OR.SHORT: "short", OR.INT: "int", OR.TIME: "time", OR.FLOAT: "float", OR.DOUBLE: "double"}


def values(rng, kind, n, npt):
    """ties: four values and a rest; spread: few repeats; edge: one class only until the last values"""
    if kind == "ties":
        x = rng.choice([3, 5, 7, 11, 0, 100, 101], n, p=[.3, .25, .2, .1, .05, .05, .05])
    elif kind == "spread":
        x = rng.integers(0, 120 if np.dtype(npt).itemsize == 1 else 30000, n)
    else:
        x = np.full(n, 42)
        x[-max(n // 50, 1):] = rng.integers(0, 100, max(n // 50, 1))
    return x.astype(npt)


@pytest.mark.parametrize("dt", list(IDS), ids=list(IDS.values()))
@pytest.mark.parametrize("path", [[OR.DICT, OR.NONE, OR.NONE], [OR.CONST, OR.NONE], [OR.PATCH, OR.NONE, OR.NONE]],
                         ids=["dict", "const", "patch"])
def test_split_and_merge_edges(G, O, rng, dt, path):
    cols, dts, trees = [], [], []
    for n in SIZES:
        for kind in ["ties", "spread", "edge"]:
            cols.append(values(rng, kind, n, OR.NP_TYPES[dt]))
            dts.append(dt)
            trees.append(G.tree_from_path(path, dt))
    run_batch(G, O, cols, dts, trees)


@pytest.mark.parametrize("dt", [OR.SHORT, OR.INT, OR.TIME], ids=["short", "int", "time"])
@pytest.mark.parametrize("path", [[OR.DICT, OR.NONE, OR.AFL, OR.NONE], [OR.CONST, OR.AFL, OR.NONE],
                                  [OR.PATCH, OR.AFL, OR.NONE, OR.AFL, OR.NONE],
                                  [OR.PATCH, OR.SCALE, OR.AFL, OR.NONE, OR.SCALE, OR.AFL, OR.NONE],
                                  [OR.DELTA, OR.CONST, OR.AFL, OR.NONE],
                                  [OR.DELTA, OR.SCALE, OR.PATCH, OR.AFL, OR.NONE, OR.AFL, OR.NONE]],
                         ids=["dict", "const", "patch", "patch-scale", "delta-const", "delta-scale-patch"])
def test_split_and_merge_through_views(G, O, rng, dt, path):
    """sources read through delta / scale views, decoded values unpacked from AFL streams in place"""
    cols, dts, trees = [], [], []
    for n in SIZES[1:]:
        for kind in ["ties", "spread", "edge"]:
            cols.append(values(rng, kind, n, OR.NP_TYPES[dt]))
            dts.append(dt)
            trees.append(G.tree_from_path(path, dt))
    run_batch(G, O, cols, dts, trees)


def frequent(rng, kind, n, npt):
    """columns whose most frequent values are hard to tell: equal (many values of one frequency), unique,
    few (fewer than four), marks (the values that the histogram tables use as empty marks), nans (float:
    NaNs of many payloads beside three values, so that one of them is the fourth)"""
    bits = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[np.dtype(npt).itemsize]
    if kind == "equal":
        return (np.arange(n) % 300).astype(npt)
    if kind == "unique":
        return rng.permutation(n).astype(npt)
    if kind == "few":
        return rng.choice([7, 9], n).astype(npt)
    if kind == "marks":
        marks = np.array([0x8f1b5c37a4d96e21, 0xe3779a4d51c2b867, 0xffffffffffffffff, 0, 5], np.uint64)
        with np.errstate(over="ignore"):
            return marks.astype(bits)[rng.choice(5, n, p=[.3, .25, .2, .15, .1])].view(npt)
    x = rng.choice([1, 2, 4], n).astype(npt)
    if np.issubdtype(npt, np.floating):
        pos = rng.random(n) < 0.4
        exp, man = (0x7ff << 52, 52) if bits is np.uint64 else (0xff << 23, 23)
        pay = rng.integers(1, 1 << man, n, dtype=np.uint64) | np.uint64(exp)
        sign = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(8 * np.dtype(npt).itemsize - 1)
        x.view(bits)[pos] = (pay | sign)[pos].astype(bits)
    return x


@pytest.mark.parametrize("dt", list(IDS), ids=list(IDS.values()))
def test_most_frequent_values(G, O, rng, dt):
    """dictionary and const nodes: candidates proven by the bounds, and the full histogram where not"""
    cols, dts, trees = [], [], []
    for n in [3, 2047, 2048, 2049, 4097, 40001, 300001]:
        for kind in ["equal", "unique", "few", "marks", "nans"]:
            for path in [[OR.DICT, OR.NONE, OR.NONE], [OR.CONST, OR.NONE]]:
                cols.append(frequent(rng, kind, n, OR.NP_TYPES[dt]))
                dts.append(dt)
                trees.append(G.tree_from_path(path, dt))
    run_batch(G, O, cols, dts, trees, steps=2)


@pytest.mark.parametrize("dt", list(IDS), ids=list(IDS.values()))
def test_delta_edges(G, O, rng, dt):
    """delta decode around its 1024-value units, 8192-value tiles and 64-tile groups, from plain and packed
    differences of several widths"""
    paths = [[OR.DELTA, OR.NONE], [OR.DELTA, OR.DELTA, OR.NONE]]
    if dt not in (OR.FLOAT, OR.DOUBLE):
        paths += [[OR.DELTA, OR.AFL, OR.NONE], [OR.DELTA, OR.SCALE, OR.AFL, OR.NONE]]
    cols, dts, trees = [], [], []
    for n in [1, 2, 33, 127, 128, 129, 1023, 1024, 1025, 1026, 8192, 8193, 8194, 70000, 64 * 8192 + 1, 64 * 8192 + 1030]:
        for bits in [1, 6, 12, 30]:
            if n > 70000 and bits in (6, 30):
                continue
            x = 1000 + np.cumsum(rng.integers(0, 1 << bits, n))
            cols.append((x % 97 if OR.NP_TYPES[dt] == np.int8 else x).astype(OR.NP_TYPES[dt]))
            dts.append(dt)
            trees.append(G.tree_from_path(paths[(n + bits) % len(paths)], dt))
    run_batch(G, O, cols, dts, trees)


@pytest.mark.parametrize("dt", [OR.CHAR, OR.SHORT, OR.INT, OR.TIME], ids=["char", "short", "int", "time"])
def test_pack_edges(G, O, rng, dt):
    """AFL packing around its 512-value units and 4096-value tiles, of every kind of width, read plainly and
    through views"""
    w = 8 * np.dtype(OR.NP_TYPES[dt]).itemsize
    cols, dts, trees = [], [], []
    for n in [1, 31, 511, 512, 513, 4095, 4096, 4097, 12289, 50001]:
        for bits in sorted({1, 2, 3, 5, 7, w // 4, w // 4 + 1, w // 2, w // 2 + 1, w - 1, w}):
            for path in [[OR.AFL, OR.NONE], [OR.SCALE, OR.AFL, OR.NONE], [OR.DELTA, OR.AFL, OR.NONE]]:
                if n > 5000 and bits not in (1, 5, w // 2 + 1, w):
                    continue
                x = rng.integers(0, 1 << min(bits, 62), n, dtype=np.int64)
                cols.append((-x if bits == w else x).astype(OR.NP_TYPES[dt]))
                dts.append(dt)
                trees.append(G.tree_from_path(path, dt))
    run_batch(G, O, cols, dts, trees)
