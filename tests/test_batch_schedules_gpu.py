"""The persistent schedule is prepared when a batch first chooses it: at any time in the batch's life, from
any thread, and while the calling thread has a capture of its own under way."""
import threading

import numpy as np
import pytest

import oracle as OR
from test_batch_gpu import framed_blobs

pytestmark = pytest.mark.gpu

TREES = [[OR.DELTA, OR.SCALE, OR.AFL, OR.NONE], [OR.DICT, OR.NONE, OR.AFL, OR.NONE], [OR.RLE, OR.AFL, OR.NONE, OR.NONE],
         [OR.SCALE, OR.PATCH, OR.AFL, OR.NONE, OR.DELTA, OR.AFL, OR.NONE], [OR.NONE]]


def table(G, rng, sizes=(1, 5000, 40_000)):
    cols, trees = [], []
    for path in TREES:
        for n in sizes:
            cols.append(np.repeat(rng.integers(0, 300, n // 3 + 1), 3)[:n].astype(np.int32))
            trees.append(G.tree_from_path(path, OR.INT))
    b = G.Batch(devs := [G.to_device(x) for x in cols], [OR.INT] * len(cols), trees, G.Stream())
    b.keep = devs  # the batch reads its columns where they are
    return cols, trees, b


def step(G, b, cols):
    b.compress()
    b.status()
    p, nb, framed, blobs = framed_blobs(G, b)
    outs = [G.alloc(x.nbytes) for x in cols]
    b.decompress(p, nb, outs)
    b.status()
    for x, o in zip(cols, outs):
        assert G.to_host(o).tobytes() == x.tobytes()
    return framed, blobs


def test_schedules_in_turn(G, O, rng):
    cols, trees, b = table(G, rng)
    first, blobs = step(G, b, cols)
    for x, t, blob in zip(cols, trees, blobs):
        assert np.array_equal(blob, O.tree_compress(t, x)), G.tree_names(t)
    for persistent in (True, False, True, True, False):
        b.set_schedule(persistent)
        assert np.array_equal(step(G, b, cols)[0], first)


def test_schedule_chosen_in_another_thread(G, O, rng):
    cols, _, b = table(G, rng)
    t = threading.Thread(target=b.set_schedule, args=(True,))
    t.start()
    t.join()
    assert b.schedule() == "persistent"
    persistent = step(G, b, cols)[0]
    b.set_schedule(False)
    assert np.array_equal(step(G, b, cols)[0], persistent)


def test_schedule_chosen_during_a_capture(G, O, rng):
    torch = pytest.importorskip("torch")
    cols, _, b = table(G, rng)
    first, _ = step(G, b, cols)
    x = torch.zeros(1000, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x += 1
        b.set_schedule(True)
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 2).all())
    assert np.array_equal(step(G, b, cols)[0], first)
