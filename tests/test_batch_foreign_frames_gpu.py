"""Frames that parse but belong to another batch: the same trees over longer columns.  The step reports
them (or, where the reference's empty-input rule gives an empty column, accepts them), and nothing of
another column in the batch is touched: it decodes bit for bit beside them."""
import struct

import numpy as np
import pytest

import oracle as OR
from test_batch_gpu import framed_blobs

pytestmark = pytest.mark.gpu

SPLITS = {"const": [OR.CONST, OR.NONE], "patch": [OR.PATCH, OR.NONE, OR.NONE], "dict": [OR.DICT, OR.NONE, OR.NONE]}


def frame(blobs):
    return np.concatenate([np.array([len(blobs)] + [b.size for b in blobs], np.uint64).view(np.uint8)] + list(blobs))


def compressed(G, cols, trees):
    b = G.Batch(devs := [G.to_device(x) for x in cols], [OR.INT] * len(cols), trees, G.Stream())
    b.keep = devs  # the batch reads its columns where they are
    b.compress()
    b.status()
    return b, framed_blobs(G, b)[3]


@pytest.mark.parametrize("long", [30_000, 131_072, 200_000])
@pytest.mark.parametrize("kind", list(SPLITS))
def test_stencil_of_a_longer_column(G, O, rng, kind, long):
    """A split node's stencil counts units that its column does not hold.  The healthy column's sums of
    differences (more than one group of 64 tiles) lie behind the short column's unit prefixes."""
    trees = [G.tree_from_path(SPLITS[kind], OR.INT), G.tree_from_path([OR.DELTA, OR.NONE], OR.INT)]
    short = rng.integers(0, 9, 1000).astype(np.int32)
    healthy = np.cumsum(rng.integers(-50, 51, 700_000)).astype(np.int32)
    donor, donor_blobs = compressed(G, [rng.integers(0, 9, long).astype(np.int32), healthy], trees)
    b, good_blobs = compressed(G, [short, healthy], trees)
    bad, good = G.to_device(frame(donor_blobs)), G.to_device(frame(good_blobs))
    for persistent in (False, True):
        b.set_schedule(persistent)
        outs = [G.alloc(x.nbytes) for x in (short, healthy)]
        b.decompress(bad.ptr, bad.nbytes, outs)
        with pytest.raises(G.GtscError):
            b.status()
        if not persistent:  # (the persistent step stops waiting between passes at the first error)
            assert G.to_host(outs[1]).tobytes() == healthy.tobytes()
        b.decompress(good.ptr, good.nbytes, outs)
        b.status()
        assert G.to_host(outs[0]).tobytes() == short.tobytes()
        assert G.to_host(outs[1]).tobytes() == healthy.tobytes()


@pytest.mark.parametrize("kind", ["patch", "dict"])
def test_long_stencil_over_empty_streams(G, O, rng, kind):
    """Both streams of the split are empty: an empty column whatever the stencil says."""
    trees = [G.tree_from_path(SPLITS[kind], OR.INT), G.tree_from_path([OR.DELTA, OR.NONE], OR.INT)]
    short = rng.integers(0, 9, 1000).astype(np.int32)
    healthy = np.cumsum(rng.integers(-50, 51, 700_000)).astype(np.int32)
    b, blobs = compressed(G, [short, healthy], trees)
    stencil = b"\0" + b"\xff" * 25_000
    enc, dt = trees[0][0::2], trees[0][1::2]
    blob = struct.pack("<hhi", enc[0], dt[0], len(stencil)) + stencil
    blob += b"".join(struct.pack("<hhiq", enc[k], dt[k], 8, 0) for k in (1, 2))
    odd = G.to_device(frame([np.frombuffer(blob, np.uint8), blobs[1]]))
    for persistent in (False, True):
        b.set_schedule(persistent)
        outs = [G.alloc(x.nbytes) for x in (short, healthy)]
        b.decompress(odd.ptr, odd.nbytes, outs)
        b.status()
        assert G.to_host(outs[1]).tobytes() == healthy.tobytes()
