"""The scan pipeline (aligned device operands) at the edges of its tiles and buffers: tiles of 57344
bytes, four buffers per CTA, one CTA per SM. Sizes around one tile, a ragged 16-byte vector, as many
tiles as buffers, one and several tiles per CTA; in place and out of place, with an init, and the
unaligned operands that take the other kernel. Integers bit-exact; floats as the primitives' bound
(1e-5 / 1e-12 of the compensated fp64 result on U[0,1))."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEN = {"f32": "f32_unit", "f64": "f64_unit", "i32": "i32_pm1000", "i64": "i64_full"}
NP = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}


def sizes(es):
    t, v = 57344 // es, 16 // es
    return [2, v - 1, v + 1, t - v, t - 1, t, t + 1, 4 * t, 4 * t + 1, 148 * t + v, 148 * 4 * t + 3,
            148 * 9 * t - 1]


def check(dt, got, want, n):
    if dt[0] == "i":
        assert np.array_equal(got, want), (dt, n)
    else:
        tol = 1e-5 if dt == "f32" else 1e-12
        err = np.abs(got.astype(np.float64) - want) / np.maximum(np.abs(want), 1.0)
        assert float(err.max()) <= tol, (dt, n, float(err.max()))


@pytest.mark.parametrize("dt", list(GEN))
def test_tile_and_buffer_edges(lib, px, ox, dev, dt):
    h = px.builtin(f"scan:{dt}")
    es = np.dtype(NP[dt]).itemsize
    init = np.full(1, 5, NP[dt])
    for i, n in enumerate(sizes(es)):
        if n < 2:
            continue
        x = ox.gen(GEN[dt], 60 + i, n)
        incl = ox.scan(x)
        d = dev.put(x)
        lib.parallax_scan(h, h, d.data_ptr(), n, es)
        px.check("scan")
        check(dt, dev.get(d, NP[dt], n), incl, n)
        d, o = dev.put(x), dev.put(np.zeros_like(x))
        lib.parallax_exclusive_scan(h, h, h, d.data_ptr(), o.data_ptr(), n, es, init.ctypes.data)
        px.check("exclusive_scan")
        want = np.empty_like(incl)
        want[0] = 5
        want[1:] = incl[:-1] + init[0] if dt[0] == "f" else incl[:-1] + NP[dt](5)
        check(dt, dev.get(o, NP[dt], n), want, n)


@pytest.mark.parametrize("shift", [1, 3])
def test_unaligned_operands_agree(lib, px, ox, dev, shift):
    """The same elements at an odd element offset take the plain-load kernel: same integers."""
    n = 3 * 14336 + 5
    x = ox.gen("i32_pm1000", 77, n + shift)
    h = px.builtin("scan:i32")
    d = dev.put(x)
    lib.parallax_scan(h, h, d.data_ptr() + 4 * shift, n, 4)
    px.check("scan")
    got = dev.get(d, np.int32, n + shift)
    assert np.array_equal(got[:shift], x[:shift]) and np.array_equal(got[shift:], ox.scan(x[shift:]))
