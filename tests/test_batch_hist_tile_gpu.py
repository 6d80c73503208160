"""The histogram tile (dict / const passes) is the one that was asked for, or the one that is reported."""
import numpy as np
import pytest

import oracle as OR
from test_batch_gpu import framed_blobs

pytestmark = pytest.mark.gpu

LENGTHS = [70_001, 5_000, 300]


def make(G, rng, **kw):
    cols = [rng.integers(0, 50, n).astype(np.int32) for n in LENGTHS]
    trees = [G.tree_from_path([OR.DICT, OR.NONE, OR.NONE] if n != 5_000 else [OR.CONST, OR.NONE], OR.INT) for n in LENGTHS]
    b = G.Batch(devs := [G.to_device(x) for x in cols], [OR.INT] * len(cols), trees, G.Stream(), **kw)
    b.keep = devs  # the batch reads its columns where they are
    return b, cols, trees


def hist_blocks(b):
    return sum(blocks for name, _, _, blocks in b.profile(True) if name == "hist")


def tiles(tile):
    return sum(-(-n // tile) for n in LENGTHS)


@pytest.mark.parametrize("tile", [256, 1024, 4096, 8192, 16384, 32768])
def test_given_tile_is_used(G, O, rng, tile):
    b, cols, trees = make(G, rng, tuning=G.tuning(hist_tile=tile))
    assert b.tuning().hist_tile == tile
    b.compress()
    b.status()
    assert hist_blocks(b) == tiles(tile)
    for blob, x, t in zip(framed_blobs(G, b)[3], cols, trees):
        assert np.array_equal(blob, O.tree_compress(t, x))


def test_default_and_tuned_tiles_are_reported(G, rng):
    b, _, _ = make(G, rng)
    b.compress()
    assert b.tuning().hist_tile == 4096 and hist_blocks(b) == tiles(4096)
    rep = b.autotune()
    b.compress()
    assert rep["hist_tile"] == b.tuning().hist_tile and hist_blocks(b) == tiles(rep["hist_tile"])


@pytest.mark.parametrize("tile", [0, 128, 300, 65536])
def test_other_tiles_are_refused(G, rng, tile):
    with pytest.raises(G.GtscError):
        make(G, rng, tuning=G.tuning(hist_tile=tile))
