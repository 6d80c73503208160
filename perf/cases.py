"""Performance cases: the work a program has this library do, through the package's public calls.

listed() names the cases that are followed, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (columns in device or pinned host memory, their trees, the
batch or the pipeline), run() makes one pass and work() counts the bytes a pass cannot do without.

Four families:
  table    many columns at once through `Batch`, with the trees of the learned planner: the mixed
           workload of the benchmark (ragged lengths, int32:float32:float64 = 2:1:1, six kinds of
           column) or the tick table (timestamps, prices, volumes, symbols, flags).
  column   one long column through `Batch` with the tree of one benchmark configuration.
  tree     one column through `tree_compress` / `tree_decompress`, the reference's per-column call.
  host     a mixed table in pinned host memory through `Pipeline`, to framed output in host memory.

`op` says which direction a pass takes: "compress", "decompress" or both ("roundtrip").  Streams and
columns are bytes, so outputs are compared as whole numbers; long ones come as 8-byte words.
"""
import functools
import math

import numpy as np
import torch

import gputimeseriescompressionoptimizer_b200 as g
from gputimeseriescompressionoptimizer_b200 import workloads

TORCH_TYPES = {g.SHORT: torch.int16, g.INT: torch.int32, g.TIME: torch.int64, g.FLOAT: torch.float32,
               g.DOUBLE: torch.float64}
DTYPES = {"int16": g.SHORT, "int32": g.INT, "int64": g.TIME, "float32": g.FLOAT, "float64": g.DOUBLE}

# the trees of the benchmark configurations (pre-order) and the bits a value takes in them, about
TREES = {
    "delta-afl": ([g.DELTA, g.AFL, g.NONE], 32),
    "delta-scale-afl": ([g.DELTA, g.SCALE, g.AFL, g.NONE], 5),
    "rle-afl-afl": ([g.RLE, g.AFL, g.NONE, g.AFL, g.NONE], 1),
    "dict-afl-afl": ([g.DICT, g.AFL, g.NONE, g.AFL, g.NONE], 10.6),
    "const-afl": ([g.CONST, g.AFL, g.NONE], 1),
    "patch-afl-afl": ([g.PATCH, g.AFL, g.NONE, g.AFL, g.NONE], 32),
    "gfc": ([g.GFC, g.NONE, g.NONE], 0),
}


def listed():
    return [
        # the first half of the benchmark's flagship workload (so that three of them fit the card):
        # 256 resident columns of 4 Ki to 16 Mi values, each direction
        {"name": "mixed256_compress", "family": "table", "table": "mixed", "op": "compress", "cols": 256,
         "max_len": 1 << 24, "shape": 0xB204},
        {"name": "mixed256_decompress", "family": "table", "table": "mixed", "op": "decompress", "cols": 256,
         "max_len": 1 << 24, "shape": 0xB204},
        # one chunk of a streaming tick table, each direction
        {"name": "tick40_compress", "family": "table", "table": "tick", "op": "compress", "cols": 40,
         "rows": 1 << 20},
        {"name": "tick40_decompress", "family": "table", "table": "tick", "op": "decompress", "cols": 40,
         "rows": 1 << 20},
        # a small table, written and read back: short ragged columns, bound by launches and latency
        {"name": "short64_roundtrip", "family": "table", "table": "mixed", "op": "roundtrip", "cols": 64,
         "max_len": 1 << 16, "shape": 64},
        # single long columns, one per benchmark configuration family
        {"name": "walk_long_roundtrip", "family": "column", "kind": "walk", "type": "int32",
         "tree": "delta-scale-afl", "op": "roundtrip", "n": 1 << 26},
        {"name": "zipf_long_compress", "family": "column", "kind": "zipf", "type": "int32",
         "tree": "dict-afl-afl", "op": "compress", "n": 1 << 26},
        {"name": "outliers_long_roundtrip", "family": "column", "kind": "outliers", "type": "int32",
         "tree": "patch-afl-afl", "op": "roundtrip", "n": 1 << 26},
        {"name": "price_gfc_roundtrip", "family": "column", "kind": "price", "type": "float64", "tree": "gfc",
         "op": "roundtrip", "n": 50_000_003},
        # the per-column call: a small part (a sensor's latest values) and a large timestamp-like column
        {"name": "tree_small", "family": "tree", "kind": "walk", "type": "int32", "tree": "delta-scale-afl",
         "op": "roundtrip", "n": 10_007},
        {"name": "tree_runs_large", "family": "tree", "kind": "runs", "type": "int64", "tree": "rle-afl-afl",
         "op": "roundtrip", "n": 5_000_011},
        # columns that start and end in host memory
        {"name": "host96_compress", "family": "host", "table": "mixed", "op": "compress", "cols": 96,
         "max_len": 1 << 22, "shape": 96},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


# kinds and types that meet in earnest: (kind, type, tree)
COLUMN_DRAWS = [
    ("walk", "int32", "delta-afl"), ("walk", "int32", "delta-scale-afl"), ("walk", "int64", "delta-scale-afl"),
    ("runs", "int32", "rle-afl-afl"), ("runs", "int64", "rle-afl-afl"), ("zipf", "int32", "dict-afl-afl"),
    ("zipf", "int16", "dict-afl-afl"), ("const", "int32", "const-afl"), ("outliers", "int32", "patch-afl-afl"),
    ("price", "float32", "gfc"), ("price", "float64", "gfc"),
]


def draw(rng):
    family = rng.choice(["table", "table", "table", "column", "column", "column", "tree", "host"])
    if family == "table":
        op = rng.choice(["compress", "decompress", "roundtrip"])
        if rng.random() < 0.3:
            return {"family": family, "table": "tick", "op": op, "cols": 5 * rng.randint(1, 8),
                    "rows": _log_int(rng, 4097, 1 << 20)}
        return {"family": family, "table": "mixed", "op": op, "cols": _log_int(rng, 8, 256),
                "max_len": _log_int(rng, 1 << 14, 1 << 23), "shape": rng.randrange(1 << 20)}
    if family == "host":
        return {"family": family, "table": "mixed", "op": "compress", "cols": _log_int(rng, 8, 128),
                "max_len": _log_int(rng, 1 << 16, 1 << 22), "shape": rng.randrange(1 << 20)}
    kind, dtype, tree = rng.choice(COLUMN_DRAWS)
    if family == "column":
        return {"family": family, "kind": kind, "type": dtype, "tree": tree,
                "op": rng.choice(["compress", "decompress", "roundtrip"]), "n": _log_int(rng, 20_001, 1 << 26)}
    return {"family": family, "kind": kind, "type": dtype, "tree": tree, "op": "roundtrip",
            "n": _log_int(rng, 1_001, 1 << 23)}


# ------------------------------------------------------------------------------ columns
def _uniform(n, gen):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)


def _integers(lo, hi, n, gen):
    return torch.randint(lo, hi, (n,), generator=gen, device="cuda", dtype=torch.int64)


@functools.lru_cache(maxsize=None)
def _zipf_cdf(s=1.1, ids=5000):
    p = 1.0 / np.arange(1, ids + 1) ** s
    return torch.from_numpy(np.cumsum(p / p.sum())).cuda()


def _zipf(n, gen):
    return torch.searchsorted(_zipf_cdf(), _uniform(n, gen)).clamp_(max=4999)


def _values(kind, n, gen):
    """The benchmark's generators (workloads.py) on the GPU: float64 for prices, else int64."""
    if kind == "walk":
        return 10 ** 6 + torch.cumsum(_integers(-8, 9, n, gen), 0)
    if kind == "runs":  # geometric runs of mean 32 over 16 values, neighbours differ
        head = _uniform(n, gen) < 1 / 32
        step = _integers(1, 16, n, gen) * head
        return _integers(0, 1 << 20, 16, gen)[torch.cumsum(step, 0) % 16]
    if kind == "zipf":
        return _zipf(n, gen)
    if kind == "const":
        return _integers(0, 1 << 20, 1, gen).expand(n).contiguous()
    if kind == "outliers":
        out = _uniform(n, gen) < 0.01
        return torch.where(out, _integers(0, 1 << 31, n, gen), _integers(0, 1 << 8, n, gen))
    t = torch.arange(n, device="cuda", dtype=torch.float64)
    x = 100 * torch.sin(2 * math.pi / 1000 * t)
    x += 0.01 * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.round(100 * x) / 100


def _specials(x, gen):
    """0.1 % NaNs of random payload and sign, a few infinities and a -0.0."""
    n = x.numel()
    k = max(n // 1000, 1)
    pos = min(n // k, 1000) * torch.arange(k, device="cuda") + _integers(0, min(n // k, 1000), k, gen)
    if x.dtype == torch.float64:
        bits = _integers(1, 1 << 52, k, gen) | (0x7FF << 52) | (_integers(0, 2, k, gen) << 63)
        x.view(torch.int64)[pos] = bits
    else:
        bits = _integers(1, 1 << 23, k, gen) | (0xFF << 23) | (_integers(0, 2, k, gen) << 31)
        x.view(torch.int32)[pos] = bits.to(torch.int32)
    x[n // 3], x[n // 2], x[n - 1] = math.inf, -math.inf, -0.0


def _column(kind, dtype, n, gen):
    v = _values(kind, n, gen)
    t = TORCH_TYPES[dtype]
    if t.is_floating_point:
        x = v.to(t)
        if kind == "price":
            _specials(x, gen)
        return x
    if kind == "price":
        v = torch.round(100 * v)
    info = torch.iinfo(t)
    return v.clamp(info.min, info.max).to(t)


def _tick_column(c, rows, gen):
    kind = workloads.TICK_COLUMNS[c % len(workloads.TICK_COLUMNS)]
    if kind == "ts":  # microseconds, exponential gaps of mean 1 ms
        gaps = -1000.0 * torch.log1p(-_uniform(rows, gen))
        return 1_700_000_000_000_000 + torch.cumsum(gaps.to(torch.int64), 0)
    if kind == "price":  # a walk in cents
        start = _integers(1000, 101_000, 1, gen)
        return (start + torch.cumsum(_integers(-1, 2, rows, gen), 0)).to(torch.float64) / 100
    if kind == "volume":  # skewed lot sizes x 100
        lots = torch.floor(1.0 / (1.0 - _uniform(rows, gen)) ** 2).clamp_(max=10_000)
        return (lots.to(torch.int32) * 100).to(torch.int32)
    if kind == "symbol":
        return _zipf(rows, gen).to(torch.int32)
    if (c // len(workloads.TICK_COLUMNS)) % 4 == 0:
        return _integers(0, 16, 1, gen).expand(rows).to(torch.int32).contiguous()
    return _integers(0, 4, rows, gen).to(torch.int32)


def _specs(case):
    """[(kind, data type, values)] of the case's columns; from the case alone."""
    if case["family"] in ("column", "tree"):
        return [(case["kind"], DTYPES[case["type"]], case["n"])]
    if case["table"] == "tick":
        types = {"ts": g.TIME, "price": g.DOUBLE}
        kinds = [workloads.TICK_COLUMNS[c % len(workloads.TICK_COLUMNS)] for c in range(case["cols"])]
        return [(k, types.get(k, g.INT), case["rows"]) for k in kinds]
    cols = workloads.mixed_columns(case["cols"], seed=case["shape"], max_len=case["max_len"])
    return [(kind, dtype, n) for kind, dtype, n, _ in cols]


class _Slice:
    """A column inside a larger device or pinned buffer: what Batch and Pipeline take."""

    def __init__(self, t):
        self.t, self.ptr, self.nbytes = t, t.data_ptr(), t.numel()


def _flat(sizes, **kw):
    """One zeroed byte buffer and its 256-byte aligned pieces."""
    offs = np.cumsum([0] + [-(-max(s, 1) // 256) * 256 for s in sizes])
    flat = torch.zeros(int(offs[-1]), dtype=torch.uint8, **kw)
    return flat, [_Slice(flat[o:o + s]) for o, s in zip(offs[:-1].tolist(), sizes)]


def _columns(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    specs = _specs(case)
    _, cols = _flat([n * g.dtype_size(dt) for _, dt, n in specs], device="cuda")
    for c, (kind, dt, n) in enumerate(specs):
        tick = case.get("table") == "tick"
        x = _tick_column(c, n, gen) if tick else _column(kind, dt, n, gen)
        cols[c].t.copy_(x.view(torch.uint8))
    torch.cuda.synchronize()
    return cols, [dt for _, dt, _ in specs]


# ------------------------------------------------------------------------------ the library's side
@functools.lru_cache(maxsize=None)
def _stream():
    return g.Stream()  # the program's one compute stream


@functools.lru_cache(maxsize=None)
def _planner():
    return g.Planner.load()


def _keep(dst, ptr, nbytes):
    """Moves a compressed result into the program's own buffer, as the next pass reuses the library's."""
    g.check(g.lib().gtsc_memcpy_async(dst.data_ptr(), ptr, nbytes, 3, _stream().handle), "keep")


def _trees(case, cols, dtypes):
    if case["family"] in ("column", "tree"):
        return [g.tree_from_path(TREES[case["tree"]][0], dtypes[0])]
    return [t for t, _ in _planner().plan(cols, dtypes)]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.family, s.op = case["family"], case["op"]
    s.cols, dtypes = _columns(case, seed)
    s.trees = _trees(case, s.cols, dtypes)
    sizes = [c.nbytes for c in s.cols]
    # room for the compressed streams (GFC and AFL may grow a column a little); zero past what is written
    room = -(-(3 * sum(sizes) // 2 + 4096 * len(sizes)) // 8) * 8
    if s.family == "host":
        host, pieces = _flat(sizes, pin_memory=True)
        for p, c in zip(pieces, s.cols):
            p.t.copy_(c.t)
        s.cols, s.host = pieces, host
        s.pipe = g.Pipeline(sizes, dtypes, s.trees, groups=8)
        s.framed = torch.zeros(room, dtype=torch.uint8, pin_memory=True)
        return s
    if s.op != "decompress":
        s.framed = torch.zeros(room, dtype=torch.uint8, device="cuda")
    if s.family == "tree":
        s.back = torch.zeros(sizes[0], dtype=torch.uint8, device="cuda")
    else:
        s.batch = g.Batch(s.cols, dtypes, s.trees, _stream())
        s.flat, s.outs = _flat(sizes, device="cuda")
        if s.op == "decompress":
            s.batch.compress()
            s.ptr, s.nbytes = s.batch.output()
    torch.cuda.synchronize()
    return s


def run(s):
    if s.family == "host":
        sizes = s.pipe.compress_host([c.ptr for c in s.cols], s.framed.data_ptr(), s.framed.numel())
        return {"sizes": sizes.astype(np.int64), "framed": s.framed.view(torch.int64)}
    if s.family == "tree":
        st = _stream().handle
        s.blob = g.tree_compress(s.trees[0], s.cols[0], st)
        _keep(s.framed, s.blob.ptr, s.blob.nbytes)
        s.column, _ = g.tree_decompress(s.blob, st)
        _keep(s.back, s.column.ptr, s.column.nbytes)
        return {"blob": s.framed.view(torch.int64), "column": s.back}
    out = {}
    if s.op != "decompress":
        s.batch.compress()
        s.ptr, s.nbytes = s.batch.output()
        _keep(s.framed, s.ptr, s.nbytes)
        out["framed"] = s.framed.view(torch.int64)
    if s.op != "compress":
        s.batch.decompress(s.ptr, s.nbytes, s.outs)
        out["columns"] = s.flat.view(torch.int64)
    return out


def work(case):
    """Bytes of one pass: the columns and their compressed streams, each read or written once a
    direction.  Stream sizes are about those of the generators' values in these trees (the mixed
    workload compresses 2.56 times, the tick table 5.8 times)."""
    raw = sum(n * g.dtype_size(dt) for _, dt, n in _specs(case))
    if case["family"] in ("column", "tree"):
        bits = TREES[case["tree"]][1]
        packed = 1.06 * raw if case["tree"] == "gfc" else case["n"] * bits / 8
    else:
        packed = raw / (5.8 if case["table"] == "tick" else 2.56)
    return {"bytes": (raw + packed) * (2 if case["op"] == "roundtrip" else 1), "flops": 0}
