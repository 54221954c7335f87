"""Tile shapes of the radix digit passes, against the oracle's sort: the rows per warp grow in
steps of four with the array (256-key rows over eight warps), a full tile is 14336 4-byte or
9216 8-byte keys, and arrays of more tiles than resident CTAs (two per SM) make the persistent
CTAs take several. Sorting moves bits, so results are compared byte for byte."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP = 1024                      # keys of four rows on all warps
TILE = {4: 56 * 256, 8: 36 * 256}
RESIDENT = 2 * 148


def sizes(es):
    t = TILE[es]
    return [STEP - 1, STEP, STEP + 1, STEP * RESIDENT - 1, STEP * RESIDENT + 1,
            t * RESIDENT - 255, t * RESIDENT, t * RESIDENT + 1]


@pytest.mark.parametrize("dtype", ["u32", "f32", "i64", "f64"])
def test_row_steps_and_waves(lib, px, ox, dev, monkeypatch, dtype):
    monkeypatch.setenv("PARALLAX_SORT", "radix")
    np_t = {"u32": np.uint32, "f32": np.float32, "i64": np.int64, "f64": np.float64}[dtype]
    es = np.dtype(np_t).itemsize
    for i, n in enumerate(sizes(es)):
        x = np.frombuffer(np.random.default_rng(40 + i).bytes(n * es), np_t).copy()
        if dtype[0] == "f":  # finite values of every magnitude, both signs
            x = np.where(np.isfinite(x), x, np_t(0))
        d = dev.put(x)
        lib.parallax_sort(px.builtin(f"sort:{dtype}"), d.data_ptr(), n, es)
        px.check("parallax_sort")
        got = dev.get(d, np_t, n)
        assert np.array_equal(got.view(np.uint8), ox.sort(x).view(np.uint8)), (dtype, n)


def test_segments_of_every_tile_fill(lib, px, dev):
    """Segments of 0 and 1 records, around a row step, a tile and several tiles, sorted stably
    by key in one call."""
    t = TILE[8]
    lens = [0, 1, 2, 31, 255, 256, STEP - 1, STEP, STEP + 1, 5 * STEP + 3, t - 1, t, t + 1, 3 * t,
            0, 7 * t + 13, 1]
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    n = int(off[-1])
    keys = np.random.default_rng(9).integers(0, 700, n).astype(np.uint64)
    rec = (keys << np.uint64(32)) | np.arange(n, dtype=np.uint64)
    d, o = dev.put(rec), dev.put(off)
    st = lib.parallax_segmented_sort(px.builtin("sort_kv:u32"), d.data_ptr(), n, o.data_ptr(), len(lens))
    assert st == px.OK
    got = dev.get(d, np.uint64, n)
    for s in range(len(lens)):
        a, b = int(off[s]), int(off[s + 1])
        assert np.array_equal(got[a:b], rec[a:b][np.argsort(keys[a:b], kind="stable")]), s


@pytest.mark.parametrize("dtype", ["u32", "f64"])
def test_small_batches_use_small_tiles(lib, px, ox, dev, monkeypatch, dtype):
    """A batch of less than a tile per SM is cut into smaller tiles: segments around their size, sorted
    by the radix path."""
    monkeypatch.setenv("PARALLAX_SORT", "radix")
    np_t = {"u32": np.uint32, "f64": np.float64}[dtype]
    es = np.dtype(np_t).itemsize
    rng = np.random.default_rng(12)
    for scale in (1, 7, 30):  # 4 to 40-odd rows per warp
        lens = [0, 1, STEP - 1, STEP, STEP + 1, 100 * STEP * scale // 7 + 5, 3, 0, 2 * STEP * scale + 1]
        off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
        n = int(off[-1])
        x = rng.integers(0, 2 ** 32, n, dtype=np.uint32) if dtype == "u32" else rng.standard_normal(n)
        d, o = dev.put(x), dev.put(off)
        st = lib.parallax_segmented_sort(px.builtin(f"sort:{dtype}"), d.data_ptr(), n, o.data_ptr(), len(lens))
        assert st == px.OK
        got = dev.get(d, np_t, n)
        for s in range(len(lens)):
            a, b = int(off[s]), int(off[s + 1])
            if b > a:
                assert np.array_equal(got[a:b].view(np.uint8), ox.sort(x[a:b]).view(np.uint8)), (scale, s)
