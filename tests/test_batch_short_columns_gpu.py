"""Batches of few short columns, whose split and delta passes run as clusters of blocks, one launch each: around
the 8192-value tiles and the eight tiles of a cluster; a longer column keeps the batch's in two.  Blobs against
the oracle byte for byte, decodes bit for bit, both schedules (run_batch)."""
import numpy as np
import pytest

import oracle as OR
from test_batch_foreign_frames_gpu import compressed, frame
from test_batch_gpu import run_batch
from test_batch_tiles_gpu import values

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 33, 1025, 8191, 8192, 8193, 16385, 40001, 65535, 65536]
IDS = {OR.CHAR: "char", OR.SHORT: "short", OR.INT: "int", OR.TIME: "time", OR.FLOAT: "float", OR.DOUBLE: "double"}
SPLITS = [[OR.DICT, OR.NONE, OR.NONE], [OR.CONST, OR.NONE], [OR.PATCH, OR.NONE, OR.NONE]]
FOLDED = [[OR.PATCH, OR.AFL, OR.NONE, OR.AFL, OR.NONE], [OR.DELTA, OR.SCALE, OR.PATCH, OR.AFL, OR.NONE, OR.AFL, OR.NONE]]
DELTAS = [[OR.DELTA, OR.NONE], [OR.DELTA, OR.DELTA, OR.NONE]]
PACKED = [[OR.DELTA, OR.AFL, OR.NONE], [OR.DELTA, OR.SCALE, OR.AFL, OR.NONE]]


def names(b, compress):
    return {name for name, _, _, _ in b.profile(compress)}


@pytest.mark.parametrize("dt", list(IDS), ids=list(IDS.values()))
def test_split(G, O, rng, dt):
    whole = dt not in (OR.FLOAT, OR.DOUBLE)
    for path in SPLITS + (FOLDED if whole and dt != OR.CHAR else []):
        for kind in ["ties", "spread", "edge"]:
            cols = [values(rng, kind, n, OR.NP_TYPES[dt]) for n in (SIZES[2:] if path in FOLDED else SIZES)]
            b, _, _ = run_batch(G, O, cols, [dt] * len(cols), [G.tree_from_path(path, dt)] * len(cols), steps=2)
            assert "split_short" in names(b, True) and "split" not in names(b, True)


@pytest.mark.parametrize("dt", list(IDS), ids=list(IDS.values()))
def test_delta(G, O, rng, dt):
    whole = dt not in (OR.FLOAT, OR.DOUBLE)
    for path in DELTAS + (PACKED if whole else []):
        x = [1000 + np.cumsum(rng.integers(0, 1 << (1 + k % 12), n)) for k, n in enumerate(SIZES)]
        cols = [(v % 97 if dt == OR.CHAR else v).astype(OR.NP_TYPES[dt]) for v in x]
        b, _, _ = run_batch(G, O, cols, [dt] * len(cols), [G.tree_from_path(path, dt)] * len(cols), steps=2)
        assert "delta_short" in names(b, False) and "delta_sum" not in names(b, False)


@pytest.mark.parametrize("sizes", [[1000 + k for k in range(200)], [1000, 1001, 65_538, 65_539]], ids=["many", "longer"])
def test_two_passes(G, O, rng, sizes):
    cols = [values(rng, "ties", n, np.int32) for n in sizes]
    trees = [G.tree_from_path([OR.DELTA, OR.NONE] if n % 2 else [OR.PATCH, OR.NONE, OR.NONE], OR.INT) for n in sizes]
    b, _, _ = run_batch(G, O, cols, [OR.INT] * len(cols), trees)
    assert "split_short" not in names(b, True) and "delta_short" not in names(b, False)


@pytest.mark.parametrize("n,long", [(1000, 8193), (1000, 70_000), (8192, 65_536), (60_001, 300_000)])
def test_differences_of_a_longer_column(G, O, rng, n, long):
    """a frame of a longer column is reported, and the columns beside it decode"""
    trees = [G.tree_from_path([OR.DELTA, OR.AFL, OR.NONE], OR.INT)] * 2
    walk = [np.cumsum(rng.integers(-50, 51, m)).astype(np.int32) for m in (n, 60_000, long)]
    _, donor = compressed(G, [walk[2], walk[1]], trees)
    b, good = compressed(G, walk[:2], trees)
    bad, ok = G.to_device(frame([donor[0], good[1]])), G.to_device(frame(good))
    for persistent in (False, True):
        b.set_schedule(persistent)
        outs = [G.alloc(x.nbytes) for x in walk[:2]]
        b.decompress(bad.ptr, bad.nbytes, outs)
        with pytest.raises(G.GtscError):
            b.status()
        if not persistent:
            assert G.to_host(outs[1]).tobytes() == walk[1].tobytes()
        b.decompress(ok.ptr, ok.nbytes, outs)
        b.status()
        assert [G.to_host(o).tobytes() for o in outs] == [x.tobytes() for x in walk[:2]]
