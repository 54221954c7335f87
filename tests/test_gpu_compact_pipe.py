"""Compaction kernels by size: single sub-tiles (57344 bytes), 114688-byte tiles up to two per SM, and
beyond that the pipeline (tiles of 53760 bytes, four buffers per CTA), at the edges of each; and the
division-free x % m == r of 64-bit integers. Values are moved, so everything is compared bit for bit
with the same selection made on the host."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 148
PIPE, TILE, SUB = 53760, 114688, 57344
DT = {"i32": np.int32, "f32": np.float32, "i64": np.int64, "f64": np.float64}


def sizes(es):
    wave = 2 * SMS * TILE // es
    return [1, SUB // es - 1, SUB // es + 1, SMS // 2 * TILE // es, SMS // 2 * TILE // es + 1, wave,
            wave + 1, (wave // (PIPE // es) + 1) * (PIPE // es), 4 * SMS * PIPE // es + 16 // es + 1,
            5 * SMS * PIPE // es - 1]


def call(lib, px, dev, spec, x):
    d, o = dev.put(x), dev.put(np.zeros_like(x))
    h = px.builtin(spec)
    k = lib.parallax_copy_if(h, h, h, h, d.data_ptr(), o.data_ptr(), x.size, x.itemsize, 0)
    px.check(spec)
    return k, dev.get(o, x.dtype, x.size)


@pytest.mark.parametrize("dt", list(DT))
def test_tile_edges(lib, px, dev, dt):
    es = np.dtype(DT[dt]).itemsize
    rng = np.random.default_rng(17)
    for n in sizes(es):
        v = rng.integers(-1000, 1001, n).astype(DT[dt])
        for spec, m in ((f"copy_if:{dt}:gt:0", v > 0), (f"remove_if:{dt}:gt:0", ~(v > 0)),
                        (f"partition:{dt}:lt:0", v < 0)):
            k, got = call(lib, px, dev, spec, v)
            assert k == int(m.sum()), (spec, n)
            want = np.concatenate([v[m], v[~m]]) if spec[0] == "p" else v[m]
            assert np.array_equal(got[:want.size], want), (spec, n)
        u = np.sort(v)[::-1].copy() if n % 2 else np.sort(v)
        first = np.concatenate([[True], u[1:] != u[:-1]])
        k, got = call(lib, px, dev, f"unique:{dt}", u)
        assert k == int(first.sum()) and np.array_equal(got[:k], u[first]), n


@pytest.mark.parametrize("keep", ["all", "none", "one_end"])
def test_extreme_selections_in_place_order(lib, px, dev, keep):
    n = 3 * SMS * PIPE // 4 + 5
    v = np.arange(1, n + 1, dtype=np.int32)
    c = {"all": 0, "none": n + 1, "one_end": n - 1}[keep]
    k, got = call(lib, px, dev, f"copy_if:i32:gt:{c}", v)
    want = v[v > c]
    assert k == want.size and np.array_equal(got[:k], want)
    k, got = call(lib, px, dev, f"partition:i32:gt:{c}", v)
    assert k == want.size and np.array_equal(got, np.concatenate([want, v[v <= c]]))


MODS = [1, -1, 2, 3, -3, 10, 64, 2 ** 31 - 1, 2 ** 32, 2 ** 32 + 15, -(2 ** 40), 2 ** 62, 2 ** 63 - 1]


@pytest.mark.parametrize("dt", ["i64", "u64"])
def test_mod_64_bit(lib, px, dev, dt):
    """C's remainder (sign of x) over extremes, multiples and their neighbours, for moduli of either
    sign, powers of two and remainders of both signs, above and at the modulus."""
    lo, hi = (-(2 ** 63), 2 ** 63 - 1) if dt == "i64" else (0, 2 ** 64 - 1)
    rng = np.random.default_rng(23)
    for m in MODS:
        am = abs(m) if dt == "i64" else m % 2 ** 64
        xs = [0, 1, -1, 2, hi, hi - 1, lo, lo + 1]
        for _ in range(60):
            q = int(rng.integers(0, 2 ** 63)) % max(1, hi // am + 1)
            xs += [s * q * am + e for s in (1, -1) for e in (-2, -1, 0, 1, 2)]
        xs += [int(v) for v in rng.integers(-(2 ** 63), 2 ** 63, 200)]
        xs = [x for x in xs if lo <= x <= hi]
        v = np.array(xs, dtype=np.int64 if dt == "i64" else np.uint64)
        for r in sorted({0, 1, -1, 2, am - 1, am, -(am - 1)}):
            if not -(2 ** 63) <= r < 2 ** 63 or (dt == "u64" and r < 0):
                continue
            rem = [(abs(x) % am) * (1 if x >= 0 else -1) for x in xs]
            want = np.array([a == r for a in rem])
            k, got = call(lib, px, dev, f"copy_if:{dt}:mod:{m}:{r}", v)
            assert k == int(want.sum()) and np.array_equal(got[:k], v[want]), (dt, m, r)
