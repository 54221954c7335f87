"""What a program asks of this runtime, as cases that can be timed and compared.

Every case is one pass through the public C ABI (the ctypes binding of
libparallax-runtime.so), called the way a program calls it: operands in device memory
(torch tensors), in device-resident arena blocks, or in coherent arena blocks that the host
reads and writes; small calls and calls that return a host value synchronous, bulk calls
enqueued on the program's own stream.

listed() names one case per use; draw() gives others of the same ranges.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent

TORCH = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "i64": torch.int64,
         "u32": torch.int32, "u64": torch.int64}  # unsigned keys as their bit patterns
NUMPY = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}
SIZE = {"f32": 4, "f64": 8, "i32": 4, "i64": 8, "u32": 4, "u64": 8}


# ---- the program's side of the runtime --------------------------------------------------------
def _load():
    name = "parallax_runtime_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            name, ROOT / "parallax-runtime_b200" / "__init__.py")
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


class _Runtime:
    """The library, the program's stream and the handles it looked up once."""

    def __init__(self):
        self.px = _load()
        self.lib = self.px.load()
        self.stream = torch.cuda.Stream()
        if self.lib.parallax_set_stream(self.stream.cuda_stream) != self.px.OK:
            raise RuntimeError("parallax_set_stream failed")
        self.handles: dict[str, int] = {}
        self.is_async = False
        self.serving = False

    def handle(self, spec: str) -> int:
        if spec not in self.handles:
            self.handles[spec] = self.px.builtin(spec)
        return self.handles[spec]

    def mode(self, asynchronous: bool) -> None:
        if asynchronous != self.is_async:
            self.lib.parallax_set_async(int(asynchronous))
            self.is_async = asynchronous

    def serve(self) -> None:
        if not self.serving:
            if self.lib.parallax_serve_start(None) != self.px.OK:
                raise RuntimeError("parallax_serve_start failed")
            self.serving = True


_runtime = None


def runtime() -> _Runtime:
    global _runtime
    if _runtime is None:
        _runtime = _Runtime()
    return _runtime


class ArenaBlock:
    """An arena block that is given back when its owner goes."""

    def __init__(self, nbytes: int, resident: bool):
        rt = runtime()
        self.lib = rt.lib
        self.nbytes = nbytes
        self.ptr = rt.lib.parallax_arena_alloc(nbytes, 256)
        if not self.ptr:
            raise RuntimeError("arena allocation failed")
        if resident:
            rt.lib.parallax_arena_set_residency(self.ptr, rt.px.DEVICE_RESIDENT)

    def host(self, dtype) -> np.ndarray:
        return np.ctypeslib.as_array((C.c_ubyte * self.nbytes).from_address(self.ptr)).view(dtype)

    def device(self, dtype: torch.dtype) -> torch.Tensor:
        """The block's device memory as a tensor (valid while the block lives)."""
        class View:
            __cuda_array_interface__ = {
                "shape": (self.nbytes,), "typestr": "|u1", "version": 2,
                "data": (self.lib.parallax_arena_device_ptr(self.ptr), False)}
        return torch.as_tensor(View(), device="cuda").view(dtype)

    def __del__(self):
        if getattr(self, "ptr", None):
            self.lib.parallax_arena_free(self.ptr)


# ---- inputs ---------------------------------------------------------------------------------
def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(g: torch.Generator, dtype: str, n: int, full: bool = False) -> torch.Tensor:
    """U[0,1) floats; integers U[-1000, 1000], or over their whole range."""
    t = torch.empty(n, dtype=TORCH[dtype], device="cuda")
    if dtype in ("f32", "f64"):
        return t.uniform_(generator=g)
    if not full:
        return t.random_(-1000, 1001, generator=g)
    if SIZE[dtype] == 4:
        return t.random_(-2 ** 31, 2 ** 31, generator=g)
    return t.random_(-2 ** 63, None, generator=g)


def _keys(g: torch.Generator, dtype: str, n: int) -> torch.Tensor:
    """Sort keys: integers over their whole range; floats U[-1,1) with 1 % exact duplicates
    and both zeros."""
    k = _values(g, dtype, n, full=True)
    if dtype in ("f32", "f64"):
        k.mul_(2).sub_(1)
        m = n // 100
        k[:100 * m:100] = k[50:100 * m:100].clone()
        step = max(1, n // 4096)
        k[7::2 * step] = 0.0
        k[11::2 * step] = -0.0
    return k


def _sorted_runs(g: torch.Generator, dtype: str, n: int) -> torch.Tensor:
    """Sorted values in runs of geometric length (mean 4)."""
    starts = torch.empty(n, dtype=torch.float32, device="cuda").uniform_(generator=g) < 0.25
    return torch.cumsum(starts, 0, dtype=torch.int64).to(TORCH[dtype])


def _lengths(case: dict) -> np.ndarray:
    """Segment lengths: lognormal, clipped to [1, 2^22], cut off at `total` elements. They
    belong to the case, not to the seed of its values."""
    rng = np.random.default_rng(11)
    lens = np.clip(np.rint(rng.lognormal(math.log(case["median"]), case["sigma"],
                                         case["segments"])), 1, 1 << 22).astype(np.int64)
    keep = int(np.searchsorted(np.cumsum(lens), case["total"], side="right"))
    return lens[:max(1, keep)]


SERVE_MIX = (("reduce", 0.4), ("scan", 0.7), ("sort", 0.9), ("copy_if", 1.0))


def _requests(case: dict) -> list[tuple[str, str, int]]:
    """(operation, type, elements) of every request of a serving batch: 40 % reduce, 30 %
    exclusive scan, 20 % sort, 10 % copy_if, sizes log-uniform from 2^10. They belong to the
    case, not to the seed of its values."""
    r = random.Random(13)
    out = []
    for _ in range(case["requests"]):
        u = r.random()
        op = next(name for name, upto in SERVE_MIX if u < upto)
        n = int(round(2.0 ** r.uniform(10, math.log2(case["n"]))))
        out.append((op, r.choice(("f32", "f64", "i32", "i64")), n))
    return out


def _predicate(dtype: str) -> str:
    return "gt:0.5" if dtype in ("f32", "f64") else "mod:3:0"


# ---- cases ----------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # the smallest call of a program whose data lives in the arena: a synchronous sum
        # over a coherent block, where call latency is everything
        {"name": "reduce_small", "op": "reduce", "kind": "sum", "dtype": "f32", "n": 1024,
         "where": "arena", "sync": True},
        # an ordinary call of the benchmark's plain configuration: synchronous in-place
        # inclusive scan of 2^20 integers in device memory
        {"name": "scan_1m", "op": "scan", "dtype": "i32", "n": 1 << 20, "sync": True},
        # a bulk reduction enqueued on the program's stream, result on the device
        {"name": "reduce_large", "op": "reduce", "kind": "sum", "dtype": "f32", "n": 1 << 28,
         "where": "device", "sync": False},
        # the largest single-array scan of the benchmark
        {"name": "exclusive_scan_large", "op": "exclusive_scan", "dtype": "f32", "n": 1 << 28,
         "sync": False},
        # the benchmark's largest 4-byte sort (out of place: the program keeps its keys)
        {"name": "sort_large", "op": "sort", "dtype": "u32", "n": 1 << 26, "sync": False},
        # a sort of ragged, ordinary size with 8-byte floating-point keys, synchronous
        {"name": "sort_ragged", "op": "sort", "dtype": "f64", "n": 700_001, "sync": True},
        # the benchmark's largest filter; returns the kept count, so it is synchronous
        {"name": "copy_if_large", "op": "copy_if", "dtype": "i32", "n": 1 << 28, "sync": True},
        # stable partition of an odd-sized array by sign
        {"name": "partition_ragged", "op": "partition", "dtype": "i32", "n": 33_554_467,
         "sync": True},
        # the batched configuration: reduce, exclusive scan and filter over 4096 uneven
        # segments of one array
        {"name": "segmented_mix", "op": "segmented", "dtype": "f32", "segments": 4096,
         "median": 4096, "sigma": 2.0, "total": 1 << 28, "sync": False},
        # the batched configuration's key-value sort (u32 keys, u32 values)
        {"name": "segmented_sort_kv", "op": "segmented_sort_kv", "segments": 4096,
         "median": 4096, "sigma": 2.0, "total": 1 << 28, "sync": False},
        # records with stored arena pointers: map with a capture and in-kernel relocation,
        # then a sum of its output
        {"name": "map_reduce", "op": "map_reduce", "n": 1 << 24, "sync": False},
        # a batch of small and ordinary requests through the serving loop
        {"name": "serve_batch", "op": "serve", "requests": 64, "n": 1 << 20},
    ]


def draw(rng: random.Random) -> dict:
    def size(lo: int, hi: int) -> int:
        """Log-uniform between powers of two, mostly odd."""
        n = int(round(2.0 ** rng.uniform(lo, hi)))
        return n | 1 if rng.random() < 0.75 else n

    op = rng.choice(("reduce", "reduce", "scan", "exclusive_scan", "exclusive_scan", "sort",
                     "sort", "copy_if", "remove_if", "partition", "unique", "segmented",
                     "segmented_sort_kv", "map_reduce", "serve"))
    dtype = rng.choice(("f32", "f64", "i32", "i64"))
    wide = 1 if SIZE[dtype] == 8 else 0
    if op == "reduce":
        n = size(10, 28 - wide)
        where = "arena" if n <= 1 << 16 and rng.random() < 0.5 else "device"
        return {"op": op, "kind": rng.choice(("sum", "sum", "max", "min")), "dtype": dtype, "n": n,
                "where": where, "sync": where == "arena" or n < 1 << 22 or rng.random() < 0.5}
    if op in ("scan", "exclusive_scan"):
        n = size(10, 28 - wide)
        return {"op": op, "dtype": dtype, "n": n, "sync": n < 1 << 22 or rng.random() < 0.5}
    if op == "sort":
        dtype = rng.choice(("u32", "i32", "f32", "u64", "i64", "f64", "kv"))
        n = size(10, 26 if dtype in ("u32", "i32", "f32") else 25)
        return {"op": op, "dtype": dtype, "n": n, "sync": n < 1 << 22 or rng.random() < 0.5}
    if op in ("copy_if", "remove_if", "partition", "unique"):
        return {"op": op, "dtype": dtype, "n": size(10, 28 - wide), "sync": True}
    if op in ("segmented", "segmented_sort_kv"):
        case = {"op": op, "segments": int(2.0 ** rng.uniform(6, 13)),
                "median": int(2.0 ** rng.uniform(6, 14)), "sigma": round(rng.uniform(0.5, 2.0), 2),
                "total": 1 << (26 - wide), "sync": rng.random() < 0.5}
        return {**case, "dtype": dtype} if op == "segmented" else case
    if op == "map_reduce":
        return {"op": op, "n": size(12, 24), "sync": rng.random() < 0.5}
    return {"op": "serve", "requests": rng.randint(16, 128), "n": 1 << rng.randint(13, 21)}


# ---- states ---------------------------------------------------------------------------------
class State:
    """One case's operands and call."""


def prepare(case: dict, seed: int) -> State:
    rt = runtime()
    s = State()
    s.case = dict(case)
    s.asynchronous = not case.get("sync", True)
    g = _generator(seed)
    globals()["_prepare_" + ("compact" if case["op"] in COMPACT else case["op"])](rt, s, case, g)
    torch.cuda.synchronize()
    return s


def run(s: State):
    rt = runtime()
    rt.mode(s.asynchronous)
    return s.call()


def _prepare_reduce(rt, s, case, g):
    dt, n = case["dtype"], case["n"]
    h = rt.handle(f"reduce:{case['kind']}:{dt}")
    x = _values(g, dt, n)
    s.x = x
    if case["where"] == "arena":
        s.block = ArenaBlock(n * SIZE[dt], resident=False)
        s.block.host(NUMPY[dt])[:] = x.cpu().numpy()
        ptr = s.block.ptr
    else:
        ptr = x.data_ptr()
    if s.asynchronous:
        s.result = torch.zeros(1, dtype=TORCH[dt], device="cuda")
        out = s.result.data_ptr()
    else:
        s.result = np.zeros(1, NUMPY[dt])
        out = s.result.ctypes.data

    def call():
        rt.lib.parallax_reduce(h, ptr, n, SIZE[dt], out)
        return {"result": s.result}
    s.call = call


def _prepare_scan(rt, s, case, g):
    """In place. Integer sums wrap, so a further pass scans what the last one left; floats
    would grow without bound, so the program scans a fresh copy each time."""
    dt, n = case["dtype"], case["n"]
    h = rt.handle(f"scan:{dt}")
    s.x = _values(g, dt, n)
    fresh = dt in ("f32", "f64")
    s.work = torch.empty_like(s.x) if fresh else s.x
    ptr = s.work.data_ptr()

    def call():
        if fresh:
            with torch.cuda.stream(rt.stream):
                s.work.copy_(s.x, non_blocking=True)
        rt.lib.parallax_scan(h, h, ptr, n, SIZE[dt])
        return {"out": s.work}
    s.call = call


def _prepare_exclusive_scan(rt, s, case, g):
    dt, n = case["dtype"], case["n"]
    h = rt.handle(f"scan:{dt}")
    s.x = _values(g, dt, n)
    s.out = torch.empty_like(s.x)
    s.init = np.full(1, 7, NUMPY[dt])
    a, b, i = s.x.data_ptr(), s.out.data_ptr(), s.init.ctypes.data

    def call():
        rt.lib.parallax_exclusive_scan(h, h, h, a, b, n, SIZE[dt], i)
        return {"out": s.out}
    s.call = call


def _prepare_sort(rt, s, case, g):
    """The runtime sorts in place; the program keeps its keys and sorts a copy."""
    kv = case["dtype"] == "kv"
    dt, n = "u64" if kv else case["dtype"], case["n"]
    h = rt.handle("sort_kv:u32" if kv else f"sort:{dt}")
    s.keys = _keys(g, dt, n)
    s.work = torch.empty_like(s.keys)
    ptr = s.work.data_ptr()

    def call():
        with torch.cuda.stream(rt.stream):
            s.work.copy_(s.keys, non_blocking=True)
        rt.lib.parallax_sort(h, ptr, n, SIZE[dt])
        return {"out": s.work}
    s.call = call


COMPACT = ("copy_if", "remove_if", "partition", "unique")


def _prepare_compact(rt, s, case, g):
    op, dt, n = case["op"], case["dtype"], case["n"]
    if op == "unique":
        s.x, spec = _sorted_runs(g, dt, n), f"unique:{dt}"
    elif op == "partition":
        s.x = _values(g, dt, n, full=True)
        if dt in ("f32", "f64"):
            s.x.sub_(0.5)
        spec = f"partition:{dt}:lt:0"
    else:
        s.x, spec = _values(g, dt, n), f"{op}:{dt}:{_predicate(dt)}"
    h = rt.handle(spec)
    s.out = torch.zeros_like(s.x)
    a, b, is_float = s.x.data_ptr(), s.out.data_ptr(), int(dt in ("f32", "f64"))

    def call():
        k = rt.lib.parallax_copy_if(h, h, h, h, a, b, n, SIZE[dt], is_float)
        return {"count": k, "out": s.out}  # beyond the kept elements the zeros stay
    s.call = call


def _offsets(lens: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)).cuda()


def _prepare_segmented(rt, s, case, g):
    dt = case["dtype"]
    lens = _lengths(case)
    S, n = len(lens), int(lens.sum())
    s.off = _offsets(lens)
    s.x = _values(g, dt, n)
    s.sums = torch.zeros(S, dtype=TORCH[dt], device="cuda")
    s.scanned = torch.empty_like(s.x)
    s.kept = torch.zeros_like(s.x)
    s.counts = torch.zeros(S, dtype=torch.int64, device="cuda")
    s.init = np.zeros(1, NUMPY[dt])
    hr, hs = rt.handle(f"reduce:sum:{dt}"), rt.handle(f"scan:{dt}")
    hc = rt.handle(f"copy_if:{dt}:" + ("gt:0.5" if dt in ("f32", "f64") else "gt:0"))
    x, off = s.x.data_ptr(), s.off.data_ptr()
    sums, scanned, kept = s.sums.data_ptr(), s.scanned.data_ptr(), s.kept.data_ptr()
    counts, init = s.counts.data_ptr(), s.init.ctypes.data

    def call():
        rt.lib.parallax_segmented_reduce(hr, x, n, off, S, sums)
        rt.lib.parallax_segmented_exclusive_scan(hs, x, scanned, n, off, S, init)
        rt.lib.parallax_segmented_copy_if(hc, x, kept, n, off, S, counts)
        return {"sums": s.sums, "scanned": s.scanned, "kept": s.kept, "counts": s.counts}
    s.call = call


def _prepare_segmented_sort_kv(rt, s, case, g):
    lens = _lengths(case)
    S, n = len(lens), int(lens.sum())
    s.off = _offsets(lens)
    s.records = torch.empty(n, dtype=torch.int64, device="cuda").random_(-2 ** 31, 2 ** 31, generator=g)
    s.records <<= 32
    start = torch.repeat_interleave(s.off[:-1], s.off[1:] - s.off[:-1])
    s.records |= torch.arange(n, device="cuda") - start
    del start
    s.work = torch.empty_like(s.records)
    h = rt.handle("sort_kv:u32")
    ptr, off = s.work.data_ptr(), s.off.data_ptr()

    def call():
        with torch.cuda.stream(rt.stream):
            s.work.copy_(s.records, non_blocking=True)
        rt.lib.parallax_segmented_sort(h, ptr, n, off, S)
        return {"out": s.work}
    s.call = call


def _prepare_map_reduce(rt, s, case, g):
    n = case["n"]
    s.target = ArenaBlock(4 * n, resident=True)
    s.records = ArenaBlock(16 * n, resident=True)
    s.y = ArenaBlock(4 * n, resident=True)
    s.target.device(torch.float32).copy_(_values(g, "f32", n))
    rec = s.records.device(torch.int64).view(n, 2)
    x = _values(g, "f32", n)
    s.at = torch.randint(n, (n,), generator=g, device="cuda")
    rec[:, 0] = x.view(torch.int32).to(torch.int64) & 0xffffffff
    rec[:, 1] = s.at * 4 + s.target.ptr
    s.x = x
    s.capture = np.array([1.5], np.float32)
    s.out = s.y.device(torch.float32)
    hm, hr = rt.handle("map:saxpy_gather_f32"), rt.handle("reduce:sum:f32")
    if s.asynchronous:
        s.result = torch.zeros(1, dtype=torch.float32, device="cuda")
        res = s.result.data_ptr()
    else:
        s.result = np.zeros(1, np.float32)
        res = s.result.ctypes.data
    records, y, cap = s.records.ptr, s.y.ptr, s.capture.ctypes.data

    def call():
        rt.lib.parallax_kernel_launch_transform2_captures(hm, records, y, n, 16, 4, cap, 4)
        rt.lib.parallax_reduce(hr, y, n, 4, res)
        return {"y": s.out, "sum": s.result}
    s.call = call


def _prepare_serve(rt, s, case, g):
    rt.serve()
    reqs = _requests(case)
    s.asynchronous = False
    s.x, s.out, s.sorted, s.keys = {}, {}, {}, {}
    s.sums = {}
    at = {k: {} for k in ("in", "sort", "sum")}
    place = []
    for op, dt, n in reqs:  # every request's operands, 256-byte aligned in one array per type
        kind = "sort" if op == "sort" else "in"
        o = at[kind].get(dt, 0)
        r = at["sum"].get(dt, 0)
        place.append((o, r))
        at[kind][dt] = o + (n + 63) // 64 * 64
        if op == "reduce":
            at["sum"][dt] = r + 1
    for dt, n in at["in"].items():
        s.x[dt] = _values(g, dt, n)
        s.out[dt] = torch.zeros_like(s.x[dt])
    for dt, n in at["sort"].items():
        s.keys[dt] = _keys(g, dt, n)
        s.sorted[dt] = torch.empty_like(s.keys[dt])
    for dt, n in at["sum"].items():
        s.sums[dt] = np.zeros(n, NUMPY[dt])
    s.counts = np.zeros(len(reqs), np.int64)
    s.requests, s.cuts = [], []
    for i, ((op, dt, n), (o, r)) in enumerate(zip(reqs, place)):
        q = rt.px.Request()
        q.count = n
        if op == "sort":
            q.kernel = rt.handle(f"sort:{dt}")
            q.input = s.sorted[dt].data_ptr() + o * SIZE[dt]
        else:
            q.input = s.x[dt].data_ptr() + o * SIZE[dt]
        if op == "reduce":
            q.kernel = rt.handle(f"reduce:sum:{dt}")
            q.result = s.sums[dt].ctypes.data + r * SIZE[dt]
        if op in ("scan", "copy_if"):
            q.output = s.out[dt].data_ptr() + o * SIZE[dt]
        if op == "scan":
            q.kernel = rt.handle(f"scan:{dt}")
            q.flags = rt.px.REQ_EXCLUSIVE
        if op == "copy_if":
            q.kernel = rt.handle(f"copy_if:{dt}:{_predicate(dt)}")
            q.result = s.counts.ctypes.data + 8 * i
        s.requests.append(q)
        s.cuts.append((op, dt, o, n))
    refs = [C.byref(q) for q in s.requests]
    tickets = [C.c_uint64() for _ in refs]
    ticket_refs = [C.byref(t) for t in tickets]

    def call():
        if s.keys:
            with torch.cuda.stream(rt.stream):
                for dt, k in s.keys.items():
                    s.sorted[dt].copy_(k, non_blocking=True)
            rt.stream.synchronize()  # the serving loop has streams of its own
        for q, t in zip(refs, ticket_refs):
            rt.lib.parallax_serve_submit(q, t)
        for t in tickets:
            rt.lib.parallax_serve_wait(t.value, None)
        # kept runs and scans share their type's output array, each at its request's place
        return {"sums": s.sums, "out": s.out, "sorted": s.sorted, "counts": s.counts}
    s.call = call


# ---- work -----------------------------------------------------------------------------------
def _kept_share(op: str, dtype: str) -> float:
    if op == "partition":
        return 1.0
    if op == "unique":
        return 0.25
    share = 0.5 if dtype in ("f32", "f64") else 667 / 2001
    return 1 - share if op == "remove_if" else share


def work(case: dict) -> dict:
    """Bytes a pass cannot do without (every input read once, every output written once) and
    its additions or comparisons."""
    op = case["op"]
    if op == "serve":
        total = flops = 0.0
        for o, dt, n in _requests(case):
            out = {"reduce": 0.0, "scan": 1.0, "sort": 1.0, "copy_if": _kept_share("copy_if", dt)}[o]
            total += n * SIZE[dt] * (1 + out)
            flops += n
        return {"bytes": total, "flops": flops}
    if op == "map_reduce":  # 16-byte record, gathered target and y; y is summed as it is made
        return {"bytes": 24 * case["n"], "flops": 3 * case["n"]}
    if op == "segmented_sort_kv":
        n = int(_lengths(case).sum())
        return {"bytes": 16 * n, "flops": n}
    if op == "segmented":  # three calls: sums; scan; filter
        n = int(_lengths(case).sum())
        return {"bytes": n * SIZE[case["dtype"]] * (1 + 2 + 1.5), "flops": 3 * n}
    n, size = case["n"], 8 if case["dtype"] == "kv" else SIZE[case["dtype"]]
    if op == "reduce":
        return {"bytes": n * size, "flops": n}
    if op in COMPACT:
        return {"bytes": n * size * (1 + _kept_share(op, case["dtype"])), "flops": n}
    return {"bytes": 2 * n * size, "flops": n}


# ---- what 64-bit arithmetic gives -------------------------------------------------------------
def exact(case: dict, seed: int):
    op = case["op"]
    g = _generator(seed)
    if op == "map_reduce":
        n = case["n"]
        target = _values(g, "f32", n).double()
        x = _values(g, "f32", n).double()
        y = 1.5 * x + target[torch.randint(n, (n,), generator=g, device="cuda")]
        return {"y": y, "sum": y.sum().reshape(1)}
    if op == "serve":
        return _exact_serve(case, g)
    dt = case.get("dtype")
    if dt not in ("f32", "f64"):
        return None
    if op == "segmented":
        lens = _lengths(case)
        off = _offsets(lens)
        x = _values(g, dt, int(lens.sum()))
        d = x.double()
        c = torch.cumsum(d, 0)
        before = torch.cat([c.new_zeros(1), c])
        sums = before[off[1:]] - before[off[:-1]]
        scanned = before[:-1] - torch.repeat_interleave(before[off[:-1]], off[1:] - off[:-1])
        return {"sums": sums, "scanned": scanned, "kept": None, "counts": None}
    if op == "reduce":
        x = _values(g, dt, case["n"])
        r = {"sum": lambda: x.double().sum(), "max": lambda: x.max(), "min": lambda: x.min()}
        return {"result": r[case["kind"]]().double().reshape(1)}
    if op == "scan":
        return {"out": torch.cumsum(_values(g, dt, case["n"]).double(), 0)}
    if op == "exclusive_scan":
        c = torch.cumsum(_values(g, dt, case["n"]).double(), 0).roll(1)
        c[0] = 0.0
        return {"out": c + 7.0}
    if op == "sort":
        return {"out": torch.sort(_keys(g, dt, case["n"])).values.double()}
    return None  # compaction moves values: nothing is computed


def _exact_serve(case: dict, g: torch.Generator):
    reqs = _requests(case)
    used = {"in": {}, "sort": {}}
    for op, dt, n in reqs:
        kind = "sort" if op == "sort" else "in"
        rows = used[kind].setdefault(dt, [])
        start = rows[-1][1] + (rows[-1][2] + 63) // 64 * 64 if rows else 0
        rows.append((op, start, n))
    sums, out, sorted_ = {}, {}, {}
    for dt, rows in used["in"].items():
        x = _values(g, dt, rows[-1][1] + (rows[-1][2] + 63) // 64 * 64)
        if dt not in ("f32", "f64"):
            if any(op == "reduce" for op, _, _ in rows):
                sums[dt] = None
            out[dt] = None
            continue
        y = torch.zeros_like(x, dtype=torch.float64)
        r = []
        for op, o, n in rows:
            v = x[o:o + n]
            if op == "reduce":
                r.append(v.double().sum())
            elif op == "scan":
                y[o + 1:o + n] = torch.cumsum(v.double(), 0)[:-1]
            else:
                k = v[v > 0.5]
                y[o:o + k.numel()] = k.double()
        if r:
            sums[dt] = torch.stack(r)
        out[dt] = y
    for dt, rows in used["sort"].items():
        k = _keys(g, dt, rows[-1][1] + (rows[-1][2] + 63) // 64 * 64)
        if dt not in ("f32", "f64"):
            sorted_[dt] = None
            continue
        y = k.double()
        for _, o, n in rows:
            y[o:o + n] = torch.sort(k[o:o + n]).values.double()
        sorted_[dt] = y
    return {"sums": sums, "out": out, "sorted": sorted_, "counts": None}
