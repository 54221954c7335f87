"""The pipeline for reduces of long segments, taken for every segment length by a tuner file that names
its shape: lengths around a work item (14332 / 7166 elements) and around a warp's part of it (896 / 448),
empty and one-element segments, starts at every element phase, segments of only the type's lowest (or
highest) value and of infinities, fewer work items than CTAs and many more. Integers and extremes
bit-exact; sums are accumulated in fp64, so fp32 results lie within one rounding (2^-23) of the fp64 sum
and fp64 ones, over chains of under 60 additions of positive terms, within 1e-14. Runs in a process of
its own, because the tuner reads its file once."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
NP = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}


def lengths(es: int, big: bool) -> list[int]:
    item, part = 57344 // es - 16 // es, 3584 // es
    some = [0, 1, 3, 7, item - 1, item, item + 1, 0, 2 * item + 5, part - 1, part, part + 1, 5, 1000, 1, 2]
    return some + ([31 * item + 3, 0, 40 * item] * 6 + [17] * 700 if big else [])


def run_checks() -> None:
    import torch

    sys.path.insert(0, str(ROOT))
    import __graft_entry__ as g

    px = g._pkg()
    lib = px.load()
    rng = np.random.default_rng(9)
    for dt, np_t in NP.items():
        es = np.dtype(np_t).itemsize
        lo, hi = (-np.inf, np.inf) if dt[0] == "f" else (np.iinfo(np_t).min, np.iinfo(np_t).max)
        for big in (False, True):
            lens = np.array(lengths(es, big))
            off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
            n, S = int(off[-1]), len(lens)
            seg = [slice(int(off[s]), int(off[s + 1])) for s in range(S)]
            o = torch.from_numpy(off.view(np.int64)).cuda()
            for kind in ("sum", "max", "min"):
                x = rng.integers(-1000, 1001, n).astype(np_t) if dt[0] == "i" else rng.random(n).astype(np_t)
                if kind != "sum":
                    x[seg[5]] = lo if kind == "max" else hi
                    x[seg[8]][3] = hi if kind == "max" else lo
                for shift in range(0, 16, es):
                    t = torch.zeros(x.nbytes + 64, dtype=torch.uint8, device="cuda")
                    t[shift:][: x.nbytes].copy_(torch.from_numpy(x.view(np.uint8)))
                    r = torch.full((S * es,), 77, dtype=torch.uint8, device="cuda")
                    torch.cuda.synchronize()
                    h = px.builtin(f"reduce:{kind}:{dt}")
                    assert lib.parallax_segmented_reduce(h, t.data_ptr() + shift, n, o.data_ptr(), S,
                                                         r.data_ptr()) == px.OK
                    got = r.cpu().numpy().view(np_t)
                    for i, s in enumerate(seg):
                        if lens[i] == 0:
                            assert got[i] == 0, (dt, kind, i)  # as the planner writes them
                        elif kind == "sum" and dt[0] == "f":
                            want = x[s].astype(np.float64).sum()
                            assert abs(got[i] - want) <= (2.0**-23 if dt == "f32" else 1e-14) * want, (dt, i)
                        else:
                            want = x[s].sum(dtype=np_t) if kind == "sum" else getattr(x[s], kind)()
                            assert got[i] == want, (dt, kind, i, shift)
    print("segmented reduce pipeline ok")


def test_reduce_pipeline_for_every_length(tmp_path):
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"{op} {t} {b} 512 7\n" for op in (0, 2, 4) for t in range(6) for b in range(31)))
    r = subprocess.run([sys.executable, __file__], env=dict(os.environ, PARALLAX_TUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "segmented reduce pipeline ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


if __name__ == "__main__":
    run_checks()
