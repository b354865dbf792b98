"""What a program that links this library has it do, as cases to be measured.

Every case is one call (or the copy and the in-place call) on
device-resident data through the C API of libclops.so, as a client written
against clo_sort.h / clo_scan.h / clo_rng.h makes it: the sorter, scanner
or generator is created once and kept, buffers wrap memory that the client
owns, and the work is enqueued on the client's queue. Sizes are those of
the benchmark (bench.py), of the command-line benchmarks (cli/*.c: sizes
doubled from 4 to 2^26, 262144 generator states), of the tests, and odd
ones between them.
"""
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "cl-ops_gb300"))
import clops  # noqa: E402

DEV = "cuda"

# Element types: (CloType, bytes, torch type of the same width). Unsigned
# types travel as torch's signed type of that width (the same bits).
TYPES = {
    "char": (clops.CLO_CHAR, 1, torch.int8), "uchar": (clops.CLO_UCHAR, 1, torch.uint8),
    "short": (clops.CLO_SHORT, 2, torch.int16), "ushort": (clops.CLO_USHORT, 2, torch.int16),
    "int": (clops.CLO_INT, 4, torch.int32), "uint": (clops.CLO_UINT, 4, torch.int32),
    "long": (clops.CLO_LONG, 8, torch.int64), "ulong": (clops.CLO_ULONG, 8, torch.int64),
    "half": (clops.CLO_HALF, 2, torch.float16), "float": (clops.CLO_FLOAT, 4, torch.float32),
    "double": (clops.CLO_DOUBLE, 8, torch.float64),
}
UNSIGNED = ("uchar", "ushort", "uint", "ulong")


def listed():
    return [
        # Radix sort of a couple of thousand keys: one of the many small sorts
        # of a client (a cell list, a batch of requests); latency is all.
        {"name": "sort_uint_2k", "kind": "sort", "algo": "satradix", "type": "uint",
         "n": 2000, "data": "uniform"},
        # The small benchmark configuration: 2^20 32-bit keys, radix=16.
        {"name": "sort_uint_1m", "kind": "sort", "algo": "satradix", "type": "uint",
         "n": 1 << 20, "data": "uniform"},
        # The headline configuration: 2^28 32-bit keys.
        {"name": "sort_uint_256m", "kind": "sort", "algo": "satradix", "type": "uint",
         "n": 1 << 28, "data": "uniform"},
        # Keys with their row numbers, a table's ragged length.
        {"name": "pairs_uint_uint_100k", "kind": "pairs", "type": "uint", "vtype": "uint",
         "n": 100003, "data": "uniform"},
        # 64-bit keys with 32-bit indices, the pair configuration.
        {"name": "pairs_ulong_uint_32m", "kind": "pairs", "type": "ulong", "vtype": "uint",
         "n": 1 << 25, "data": "uniform"},
        # Offsets of a few thousand variable-length records.
        {"name": "scan_uint_ulong_5k", "kind": "scan", "type": "uint", "stype": "ulong",
         "n": 5003},
        # The scan configuration's types, at a quarter of its length.
        {"name": "scan_uint_ulong_256m", "kind": "scan", "type": "uint", "stype": "ulong",
         "n": 1 << 28},
        # Floating-point keys go to the bitonic sorters (the radix sort takes
        # integers only); a length that is no power of two.
        {"name": "abitonic_float_1500k", "kind": "sort", "algo": "abitonic", "type": "float",
         "n": 1500001, "data": "uniform"},
        # The command-line benchmark's default sorter, signed keys.
        {"name": "sbitonic_int_64k", "kind": "sort", "algo": "sbitonic", "type": "int",
         "n": 1 << 16, "data": "uniform"},
        # Many segments of one buffer with log-normal lengths (the batched
        # configuration): sorted each by itself...
        {"name": "segsort_uint_80m", "kind": "segsort", "type": "uint", "n": 80000000,
         "segments": 10000, "sigma": 2.0},
        # ... and summed each by itself.
        {"name": "segscan_uint_ulong_3m", "kind": "segscan", "type": "uint", "stype": "ulong",
         "n": 3000017, "segments": 4001, "sigma": 1.5},
        # The random-number benchmark's default 262144 states, a batch of draws.
        {"name": "rng_mwc64x_256k_32", "kind": "rng", "gen": "mwc64x", "n": 262144, "draws": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["radix", "radix", "radix", "pairs", "pairs", "scan", "scan", "abitonic",
                       "abitonic", "sbitonic", "segsort", "segscan", "rng"])
    if kind == "radix":
        t = rng.choice(["uint", "uint", "uint", "ulong", "ushort", "uchar"])
        hi = {8: 1 << 26, 4: 1 << 28, 2: 1 << 28, 1: 1 << 28}[TYPES[t][1]]
        return {"kind": "sort", "algo": "satradix", "type": t, "n": _log_int(rng, 500, hi),
                "data": rng.choice(["uniform", "uniform", "zipf", "sorted"])}
    if kind == "pairs":
        return {"kind": "pairs", "type": rng.choice(["uint", "ulong"]),
                "vtype": rng.choice(["uint", "uint", "ulong"]),
                "n": _log_int(rng, 500, 1 << 25), "data": rng.choice(["uniform", "uniform", "zipf"])}
    if kind == "scan":
        t, s = rng.choice([("uint", "ulong"), ("uint", "uint"), ("int", "long"),
                           ("uchar", "uint"), ("ulong", "ulong")])
        return {"kind": "scan", "type": t, "stype": s, "n": _log_int(rng, 500, 1 << 28)}
    if kind == "abitonic":
        return {"kind": "sort", "algo": "abitonic",
                "type": rng.choice(["float", "float", "double", "int", "half", "long"]),
                "n": _log_int(rng, 500, 1 << 24), "data": "uniform"}
    if kind == "sbitonic":
        return {"kind": "sort", "algo": "sbitonic", "type": rng.choice(["int", "uint", "float"]),
                "n": _log_int(rng, 500, 1 << 20), "data": "uniform"}
    if kind in ("segsort", "segscan"):
        segs = _log_int(rng, 16, 20000)
        n = min(1 << 27, max(segs, int(segs * math.exp(rng.uniform(3.0, 9.0)))))
        case = {"kind": kind, "type": "uint", "n": n, "segments": segs,
                "sigma": round(rng.uniform(0.3, 2.0), 2)}
        if kind == "segscan":
            case["stype"] = rng.choice(["ulong", "uint"])
        else:
            case["type"] = rng.choice(["uint", "uint", "ulong"])
        return case
    n = _log_int(rng, 5000, 1 << 22)
    return {"kind": "rng", "gen": rng.choice(["lcg", "xorshift64", "xorshift128", "mwc64x",
                                              "parkmiller"]),
            "n": n, "draws": rng.randint(4, max(4, min(128, (1 << 28) // n)))}


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "rng":
        return {"bytes": n * (4 * case["draws"] + 2 * clops.RNG_SEED_SIZE[case["gen"]]), "flops": 0}
    e = TYPES[case["type"]][1]
    if kind == "pairs":
        return {"bytes": 2 * n * (e + TYPES[case["vtype"]][1]), "flops": 0}
    if kind in ("scan", "segscan"):
        b = n * (e + TYPES[case["stype"]][1])
        return {"bytes": b + (8 * (case["segments"] + 1) if kind == "segscan" else 0), "flops": 0}
    return {"bytes": 2 * n * e + (8 * (case["segments"] + 1) if kind == "segsort" else 0),
            "flops": 0}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _int_bits(g, n, dtype):
    """n uniformly random words of an integer type."""
    bits = torch.iinfo(dtype).bits
    words = torch.empty((n * bits // 8 + 7) // 8, dtype=torch.int64, device=DEV)
    words.random_(-(1 << 63), None, generator=g)
    return words.view(dtype)[:n].clone()


def _keys(case, seed, name="type"):
    """Keys of the case's type and distribution: uniform over the type (floats:
    over a million either side of zero, half: a thousand), Zipf-like ranks of
    2^20 hashed to keys, or uniform keys already in order."""
    t, n, g = case[name], case["n"], _gen(seed)
    dtype = TYPES[t][2]
    if dtype.is_floating_point:
        span = 1000.0 if t == "half" else 1e6
        return ((torch.rand(n, dtype=torch.float64, device=DEV, generator=g) * 2 - 1) * span).to(dtype)
    kind = case.get("data", "uniform")
    if kind == "zipf":
        rank = torch.exp2(torch.rand(n, dtype=torch.float32, device=DEV, generator=g) * 20).to(torch.int64)
        x = rank * 0x2545F4914F6CDD1D
        x = x ^ (x >> 29)
        return x.view(dtype)[:: 8 // TYPES[t][1]].clone()
    a = _int_bits(g, n, dtype)
    return _sorted_unsigned(a, t) if kind == "sorted" else a


def _sorted_unsigned(a, t):
    """`a` in ascending order of its unsigned bit patterns."""
    if t == "uchar":
        return torch.sort(a).values
    low = torch.iinfo(a.dtype).min
    return torch.sort(a ^ low).values ^ low


def _offsets(case, seed):
    """Log-normal segment lengths, scaled to add up to n; some segments are empty."""
    r = np.random.RandomState((seed + 77) % (1 << 32))
    w = np.exp(case["sigma"] * r.standard_normal(case["segments"]))
    off = np.zeros(case["segments"] + 1, dtype=np.int64)
    off[1:] = np.rint(np.cumsum(w) / w.sum() * case["n"])
    off[-1] = case["n"]
    return torch.from_numpy(off).to(DEV)


def _values(case, seed):
    """Scan inputs: record lengths below 256 (signed types: around zero)."""
    t, g = case["type"], _gen(seed)
    lo, hi = (-128, 128) if t == "int" else (0, 256)
    return torch.randint(lo, hi, (case["n"],), dtype=TYPES[t][2], device=DEV, generator=g)


def _states(case, seed):
    size = clops.RNG_SEED_SIZE[case["gen"]]
    s = _int_bits(_gen(seed), case["n"] * size // 4, torch.int32)
    return (s & 0x7FFFFFFF) % 2147483646 + 1 if case["gen"] == "parkmiller" else s


# ---------------------------------------------------------------- handles
_lib = {}


def _client():
    """The client's context and queue, one each for the process."""
    if not _lib:
        _lib["ctx"] = clops.Context(torch.cuda.current_device())
        _lib["q"] = clops.Queue(_lib["ctx"])
    return _lib["ctx"], _lib["q"]


class Wrapped:
    """A library buffer over a tensor's memory."""

    def __init__(self, ctx, t):
        self.t = t
        self.nbytes = t.numel() * t.element_size()
        self.h = clops.call(clops.lib.ccl_buffer_new_wrap, ctx.h, t.data_ptr(), self.nbytes)

    def __del__(self):
        clops.lib.ccl_buffer_destroy(self.h)


class State:
    def __init__(self, case):
        self.case = case
        self.ctx, self.q = _client()
        self.obj = None

    def __del__(self):
        if self.obj is not None:
            self.obj.destroy()


def prepare(case, seed):
    s = State(case)
    kind, n = case["kind"], case["n"]
    if kind in ("sort", "pairs", "segsort"):
        src = _keys(case, seed)
        s.src, s.dst = Wrapped(s.ctx, src), Wrapped(s.ctx, torch.empty_like(src))
        algo = case.get("algo", "satradix")
        opts = "radix=16" if algo == "satradix" else None
        s.obj = clops.Sorter(s.ctx, algo, TYPES[case["type"]][0], options=opts)
        if kind == "pairs":
            v = _int_bits(_gen(seed + 1), n, TYPES[case["vtype"]][2])
            s.vsrc, s.vdst = Wrapped(s.ctx, v), Wrapped(s.ctx, torch.empty_like(v))
    elif kind in ("scan", "segscan"):
        s.src = Wrapped(s.ctx, _values(case, seed))
        s.dst = Wrapped(s.ctx, torch.empty(n, dtype=TYPES[case["stype"]][2], device=DEV))
        s.obj = clops.Scanner(s.ctx, TYPES[case["type"]][0], TYPES[case["stype"]][0])
    else:
        seeds = Wrapped(s.ctx, _states(case, seed))
        torch.cuda.synchronize()  # the queue is no torch stream
        s.obj = clops.Rng(s.ctx, s.q, case["gen"], clops.CLO_RNG_SEED_EXT_DEV, n, seeds=seeds)
        s.src = seeds
        s.dst = Wrapped(s.ctx, torch.empty(case["draws"] * n, dtype=torch.int32, device=DEV))
    if kind in ("segsort", "segscan"):
        s.off = Wrapped(s.ctx, _offsets(case, seed))
    torch.cuda.synchronize()
    return s


def run(s):
    case, q = s.case, s.q
    kind, n = case["kind"], case["n"]
    q.gc()  # the events of earlier calls go back to the queue
    if kind == "sort":
        s.obj.sort_device(q, s.src, n, buf_out=s.dst)
        return s.dst.t
    if kind == "scan":
        s.obj.scan_device(q, s.src, s.dst, n)
        return s.dst.t
    if kind == "segscan":
        s.obj.scan_segmented_device(q, s.src, s.dst, s.off, case["segments"])
        return s.dst.t
    if kind == "rng":
        # The states move on with every batch, as a client's do.
        s.obj.fill(q, s.dst, case["draws"])
        return {"numbers": s.dst.t, "states": s.src.t}
    # These sort in place: the client keeps its originals and sorts a copy.
    _copy(s.src, s.dst, q)
    if kind == "segsort":
        s.obj.sort_segmented_device(q, s.dst, s.off, case["segments"])
        return s.dst.t
    _copy(s.vsrc, s.vdst, q)
    s.obj.sort_kv_device(q, s.dst, s.vdst, TYPES[case["vtype"]][0], n)
    return {"keys": s.dst.t, "values": s.vdst.t}


def _copy(a, b, q):
    clops.call(clops.lib.ccl_buffer_enqueue_copy, a.h, b.h, q.h, 0, 0, a.nbytes, None)


# ------------------------------------------------------------------ exact
def _order(a, t):
    """`a` as 64-bit words whose signed order is the unsigned order of its bits."""
    if t == "uchar":
        return a.to(torch.int64)
    if t in ("ulong", "long"):
        return a ^ torch.iinfo(torch.int64).min
    return a.to(torch.int64) & ((1 << (8 * TYPES[t][1])) - 1)


def exact(case, seed):
    kind, n, t = case["kind"], case["n"], case["type"] if "type" in case else None
    if kind == "rng":
        return None
    if kind in ("sort", "pairs", "segsort"):
        a = _keys(case, seed)
        if kind == "sort":
            if a.is_floating_point():
                return torch.sort(a.to(torch.float64)).values
            if case["algo"] == "satradix" or t in UNSIGNED:
                return _sorted_unsigned(a, t)
            return torch.sort(a).values
        if kind == "pairs":
            at = torch.sort(_order(a, t), stable=True).indices
            v = _int_bits(_gen(seed + 1), n, TYPES[case["vtype"]][2])
            return {"keys": a[at], "values": v[at]}
        off = _offsets(case, seed)
        at = torch.sort(_order(a, t), stable=True).indices
        seg = torch.searchsorted(off[1:], at, right=True).to(torch.int32)
        return a[at[torch.sort(seg, stable=True).indices]]
    x = _values(case, seed).to(torch.int64)
    sums = torch.cumsum(x, 0) - x
    if kind == "segscan":
        off = _offsets(case, seed)
        seg = torch.searchsorted(off[1:], torch.arange(n, device=DEV), right=True)
        sums = sums - sums[off[seg]]
    return sums.to(TYPES[case["stype"]][2])
