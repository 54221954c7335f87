"""The persistent pipelines of the plain scans and compactions, at sizes that reach them (more than 296 tiles of
114688 bytes): whole tiles of theirs (57344 bytes scan, 53760 compaction), one element and one 16-byte word more
or less, and selections and values where a pipeline can go wrong: nothing or everything kept, a single kept
element at either end, NaN, infinities and signed zeros, output written over the input. Moved values and integer
prefixes bit for bit, float prefixes within the tolerances of the other scan tests, all against torch."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAVE = 2 * 148 * 114688
SCAN, PIPE = 57344, 53760
NAMES = ["i32", "f32", "i64", "f64"]


def sizes(es, tile):
    wave, t, v = WAVE // es, tile // es, 16 // es
    full = (wave // t + 1) * t
    return [wave + 1, full - v, full - 1, full, full + 1, full + v, full + t // 2 + 1]


def types(torch, dt):
    return {"i32": (torch.int32, torch.int32), "f32": (torch.float32, torch.int32),
            "i64": (torch.int64, torch.int64), "f64": (torch.float64, torch.int64)}[dt]


def bits(torch, dt, t):
    return t.view(types(torch, dt)[1])


def compact(lib, px, torch, spec, x, out):
    h = px.builtin(spec)
    torch.cuda.synchronize()
    k = lib.parallax_copy_if(h, h, h, h, x.data_ptr(), out.data_ptr(), x.numel(), x.element_size(), 0)
    px.check(spec)
    return k


def same(torch, dt, got, want):
    return torch.equal(bits(torch, dt, got), bits(torch, dt, want))


@pytest.mark.parametrize("dt", NAMES)
def test_compaction_edges(lib, px, dev, dt):
    torch = dev.torch
    ty = types(torch, dt)[0]
    gen = torch.Generator(device="cuda").manual_seed(1)
    for n in sizes(4 if dt[1:] == "32" else 8, PIPE):
        x = torch.randint(-1000, 1001, (n,), device="cuda", generator=gen).to(ty)
        out = torch.empty_like(x)
        for spec, m in ((f"copy_if:{dt}:gt:0", x > 0), (f"remove_if:{dt}:ge:-3", ~(x >= -3))):
            k = compact(lib, px, torch, spec, x, out)
            want = x[m]
            assert k == want.numel() and same(torch, dt, out[:k], want), (spec, n)
        m = x < 0
        k = compact(lib, px, torch, f"partition:{dt}:lt:0", x, out)
        assert k == int(m.sum()) and same(torch, dt, out, torch.cat([x[m], x[~m]])), n
        x = torch.div(torch.arange(n, device="cuda"), 7, rounding_mode="floor").to(ty)  # runs across the tiles
        k = compact(lib, px, torch, f"unique:{dt}", x, out)
        assert k == (n + 6) // 7 and same(torch, dt, out[:k], x[::7].contiguous()), n


@pytest.mark.parametrize("dt", ["i32", "i64"])
@pytest.mark.parametrize("keep", ["all", "none", "last", "first"])
def test_compaction_extremes(lib, px, dev, dt, keep):
    torch = dev.torch
    ty = types(torch, dt)[0]
    n = sizes(4 if dt == "i32" else 8, PIPE)[-1]
    x = torch.arange(1, n + 1, device="cuda").to(ty)
    out = torch.empty_like(x)
    op, c = {"all": ("gt", 0), "none": ("gt", n), "last": ("gt", n - 1), "first": ("lt", 2)}[keep]
    m = x > c if op == "gt" else x < c
    for kind, mask in (("copy_if", m), ("remove_if", ~m)):
        out.fill_(-9)
        k = compact(lib, px, torch, f"{kind}:{dt}:{op}:{c}", x, out)
        want = x[mask]
        assert k == want.numel() and torch.equal(out[:k], want) and bool((out[k:] == -9).all()), kind
    k = compact(lib, px, torch, f"partition:{dt}:{op}:{c}", x, out)
    assert k == int(m.sum()) and torch.equal(out, torch.cat([x[m], x[~m]]))
    if keep in ("all", "first"):  # unique: every element, or one
        y = x if keep == "all" else torch.full_like(x, 5)
        k = compact(lib, px, torch, f"unique:{dt}", y, out)
        assert k == (n if keep == "all" else 1) and torch.equal(out[:k], y[:k])


@pytest.mark.parametrize("dt", NAMES)
def test_compaction_over_its_input(lib, px, dev, dt):
    """Every kept element moves to a place at or before its own, so the output may be the input."""
    torch = dev.torch
    ty = types(torch, dt)[0]
    n = sizes(4 if dt[1:] == "32" else 8, PIPE)[-1]
    gen = torch.Generator(device="cuda").manual_seed(2)
    for threshold in (0, 990, -1000):  # half, few and nearly all kept
        x = torch.randint(-1000, 1001, (n,), device="cuda", generator=gen).to(ty)
        want = x[x > threshold]
        k = compact(lib, px, torch, f"copy_if:{dt}:gt:{threshold}", x, x)
        assert k == want.numel() and same(torch, dt, x[:k], want), threshold
    x = torch.randint(0, 3, (n,), device="cuda", generator=gen).to(ty)
    first = torch.ones(n, dtype=torch.bool, device="cuda")
    first[1:] = x[1:] != x[:-1]
    want = x[first]
    k = compact(lib, px, torch, f"unique:{dt}", x, x)
    assert k == want.numel() and same(torch, dt, x[:k], want)


@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_compaction_of_special_values(lib, px, dev, dt):
    torch = dev.torch
    ty = types(torch, dt)[0]
    n = sizes(4 if dt == "f32" else 8, PIPE)[4]
    special = torch.tensor([float("nan"), -float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 0.5, -0.5,
                            torch.finfo(ty).tiny / 4, torch.finfo(ty).max, torch.finfo(ty).min],
                           dtype=ty, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = special[torch.randint(0, special.numel(), (n,), device="cuda", generator=gen)]
    out = torch.empty_like(x)
    for pred, m in (("gt:0", x > 0), ("ge:0", x >= 0), ("lt:0.5", x < 0.5), ("le:0", x <= 0),
                    ("eq:0", x == 0), ("ne:0", x != 0), ("nonzero", x != 0)):
        for kind, mask in (("copy_if", m), ("remove_if", ~m)):
            k = compact(lib, px, torch, f"{kind}:{dt}:{pred}", x, out)
            want = x[mask]
            assert k == want.numel() and same(torch, dt, out[:k], want), (kind, pred)
        k = compact(lib, px, torch, f"partition:{dt}:{pred}", x, out)
        assert k == int(m.sum()) and same(torch, dt, out, torch.cat([x[m], x[~m]])), pred
    first = torch.ones(n, dtype=torch.bool, device="cuda")
    first[1:] = ~(x[1:] == x[:-1])  # NaN equals nothing, -0 equals +0
    k = compact(lib, px, torch, f"unique:{dt}", x, out)
    want = x[first]
    assert k == want.numel() and same(torch, dt, out[:k], want)


@pytest.mark.parametrize("dt", NAMES)
def test_scan_edges(lib, px, dev, dt):
    torch = dev.torch
    ty = types(torch, dt)[0]
    h = px.builtin(f"scan:{dt}")
    init = np.full(1, 5, {"i32": np.int32, "f32": np.float32, "i64": np.int64, "f64": np.float64}[dt])
    gen = torch.Generator(device="cuda").manual_seed(4)

    def check(got, want, n):
        if dt[0] == "i":
            assert torch.equal(got, want), n
        else:
            tol = 1e-5 if dt == "f32" else 1e-12
            err = (got.double() - want).abs() / want.abs().clamp(min=1.0)
            assert float(err.max()) <= tol, (n, float(err.max()))

    for n in sizes(4 if dt[1:] == "32" else 8, SCAN):
        if dt[0] == "i":
            x = torch.randint(-1000, 1001, (n,), device="cuda", generator=gen).to(ty)
        else:
            x = torch.rand(n, dtype=ty, device="cuda", generator=gen)
        incl = torch.cumsum(x, 0, dtype=ty if dt[0] == "i" else torch.float64)
        excl = torch.cat([torch.zeros_like(incl[:1]), incl[:-1]]) + 5
        over = x.clone()
        for src, out in ((x, torch.empty_like(x)), (over, over)):  # into another array, over the input
            torch.cuda.synchronize()
            lib.parallax_exclusive_scan(h, h, h, src.data_ptr(), out.data_ptr(), n, x.element_size(),
                                        init.ctypes.data)
            px.check("exclusive_scan")
            check(out, excl, n)
        torch.cuda.synchronize()
        lib.parallax_scan(h, h, x.data_ptr(), n, x.element_size())
        px.check("scan")
        check(x, incl, n)


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("value", ["inf", "-inf", "nan"])
def test_scan_carries_infinities_and_nan_forward_only(lib, px, dev, dt, value):
    torch = dev.torch
    ty = types(torch, dt)[0]
    n = sizes(4 if dt == "f32" else 8, SCAN)[-1]
    gen = torch.Generator(device="cuda").manual_seed(6)
    for at in (n - 1, n // 2 + 3, 5):
        x = torch.rand(n, dtype=ty, device="cuda", generator=gen)
        want = torch.cumsum(x, 0, dtype=torch.float64)
        x[at] = float(value)
        torch.cuda.synchronize()
        h = px.builtin(f"scan:{dt}")
        lib.parallax_scan(h, h, x.data_ptr(), n, x.element_size())
        px.check("scan")
        err = (x[:at].double() - want[:at]).abs() / want[:at].clamp(min=1.0)
        assert float(err.max()) <= (1e-5 if dt == "f32" else 1e-12)
        tail = x[at:]
        assert bool(torch.isnan(tail).all() if value == "nan" else (tail == float(value)).all()), at
