"""Segmented pipelines on values and uses of their own: NaN, infinities and signed zeros through select, scans
that carry an infinity to the end of their segment only, extremes of segments that hold nothing but the type's
lowest or highest value, and a select written over its input. Every call takes its pipeline, by a tuner file that
names them; in a process of its own, because the tuner reads its file once. Against numpy per segment."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
LENGTHS = [13437, 1, 0, 50001, 14333, 7, 120003, 2, 26873] * 3


def run_checks() -> None:
    import torch

    sys.path.insert(0, str(ROOT))
    import __graft_entry__ as g

    px = g._pkg()
    lib = px.load()
    rng = np.random.default_rng(8)
    off = np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.uint64)
    n, S = int(off[-1]), len(LENGTHS)
    seg = [slice(int(off[s]), int(off[s + 1])) for s in range(S)]
    o = torch.from_numpy(off.view(np.int64)).cuda()
    counts = torch.zeros(S, dtype=torch.int64, device="cuda")

    def select(spec, src, dst, x, keep):
        torch.cuda.synchronize()
        assert lib.parallax_segmented_copy_if(px.builtin(spec), src.data_ptr(), dst.data_ptr(), n, o.data_ptr(),
                                              S, counts.data_ptr()) == px.OK
        got, k = dst.cpu().numpy().view(x.dtype), counts.cpu().numpy()
        word = np.uint32 if x.itemsize == 4 else np.uint64
        for i, s in enumerate(seg):
            want = x[s][keep[s]]
            assert k[i] == want.size, (spec, i)
            assert np.array_equal(got[s][: want.size].view(word), want.view(word)), (spec, i)

    for dt, t in (("f32", np.float32), ("f64", np.float64)):
        special = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 0.5, -0.5, np.finfo(t).tiny / 4,
                            np.finfo(t).max], t)
        x = special[rng.integers(0, special.size, n)]
        src, dst = torch.from_numpy(x).cuda(), torch.empty(n, dtype=torch.float32 if dt == "f32" else
                                                           torch.float64, device="cuda")
        for pred, keep in (("gt:0", x > 0), ("le:0", x <= 0), ("eq:0", x == 0), ("nonzero", x != 0)):
            select(f"copy_if:{dt}:{pred}", src, dst, x, keep)
            select(f"remove_if:{dt}:{pred}", src, dst, x, ~keep)
        x = rng.random(n).astype(t)
        src = torch.from_numpy(x).cuda()
        select(f"copy_if:{dt}:gt:0.5", src, src, x, x > 0.5)  # over its input

        at = [s.start + (s.stop - s.start) // 2 for s in seg if s.stop - s.start > 20000]
        x[at] = np.inf
        src, h = torch.from_numpy(x).cuda(), px.builtin(f"scan:{dt}")
        torch.cuda.synchronize()
        assert lib.parallax_segmented_inclusive_scan(h, src.data_ptr(), dst.data_ptr(), n, o.data_ptr(),
                                                     S) == px.OK
        got = dst.cpu().numpy()
        tol = 1e-5 if dt == "f32" else 1e-12
        for s in seg:
            want = np.cumsum(x[s], dtype=np.float64)
            fin = np.isfinite(want)
            assert np.all(np.abs(got[s][fin] - want[fin]) <= tol * np.maximum(1.0, want[fin]))
            assert np.all(got[s][~fin] == np.inf)

    for dt, t in (("f32", np.float32), ("f64", np.float64), ("i32", np.int32), ("i64", np.int64)):
        lo, hi = (-np.inf, np.inf) if dt[0] == "f" else (np.iinfo(t).min, np.iinfo(t).max)
        res = torch.zeros(S * np.dtype(t).itemsize, dtype=torch.uint8, device="cuda")
        for kind, v in (("max", lo), ("min", hi)):
            x = np.full(n, v, t)
            src = torch.from_numpy(x).cuda()
            torch.cuda.synchronize()
            assert lib.parallax_segmented_reduce(px.builtin(f"reduce:{kind}:{dt}"), src.data_ptr(), n,
                                                 o.data_ptr(), S, res.data_ptr()) == px.OK
            got = res.cpu().numpy().view(t)
            assert all(got[i] == (v if LENGTHS[i] else 0) for i in range(S)), (dt, kind)
    print("special values ok")


def test_special_values_on_the_pipelines(tmp_path):
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"{op} {t} {b} {shape}\n" for op, shape in ((0, "512 7"), (2, "512 7"), (4, "512 7"),
                                                                       (8, "1024 7"), (16, "1024 7"))
                             for t in range(6) for b in range(31)))
    r = subprocess.run([sys.executable, __file__], env=dict(os.environ, PARALLAX_TUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "special values ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


if __name__ == "__main__":
    run_checks()
