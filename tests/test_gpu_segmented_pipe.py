"""The pipelines for long segments (segmented scans and select), taken for every segment length by a
tuner file that names them: lengths around a work item (14332 / 7166 elements for scans, 13436 / 6718
for select), empty and one-element segments, starts at every 16-byte phase, outputs at another phase
than the input, in-place scans, both scan flavours. Against numpy per segment: integers and moved
values bit-exact, floats within 1e-5 / 1e-12 of fp64. Runs in a process of its own, because the tuner
reads its file once."""
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


def lengths(es: int) -> list[int]:
    scan, sel = 57344 // es - 16 // es, 53760 // es - 16 // es
    return [0, 1, 3, 7, scan - 1, scan, scan + 1, 0, 2 * scan + 5, sel - 1, sel, sel + 1, 3 * sel + 2, 5,
            1000, 9 * scan + 11, 1, 1, 2, 0, 40 * sel + 3, 33]


def run_checks() -> None:
    import torch

    sys.path.insert(0, str(ROOT))
    import __graft_entry__ as g

    px = g._pkg()
    lib = px.load()
    rng = np.random.default_rng(5)
    for dt, np_t in NP.items():
        es = np.dtype(np_t).itemsize
        lens = np.array(lengths(es) * 4)
        off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
        n, S = int(off[-1]), len(lens)
        x = rng.integers(-1000, 1001, n).astype(np_t) if dt[0] == "i" else rng.random(n).astype(np_t)
        seg = [slice(int(off[s]), int(off[s + 1])) for s in range(S)]

        def dev(nbytes, shift):
            t = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
            return t, t.data_ptr() + shift

        def put(p, a):
            h = torch.from_numpy(a.view(np.uint8))
            t, base = p
            t[base - t.data_ptr():][: h.numel()].copy_(h)

        def get(p):
            t, base = p
            return t[base - t.data_ptr():][: x.nbytes].cpu().numpy().view(np_t)

        o = torch.from_numpy(off.view(np.int64)).cuda()
        wide = np.float64 if dt[0] == "f" else np_t
        incl = np.concatenate([np.cumsum(x[s], dtype=wide) for s in seg])
        init = np.array([3], np_t)
        excl = np.concatenate([np.concatenate([[0], np.cumsum(x[s], dtype=wide)[:-1]]) + init[0]
                               if lens[i] else np.zeros(0) for i, s in enumerate(seg)]).astype(wide)

        def close(got, want, what):
            if dt[0] == "i":
                assert np.array_equal(got, want), what
            else:
                tol = 1e-5 if dt == "f32" else 1e-12
                assert np.all(np.abs(got - want) <= tol * np.maximum(1.0, np.abs(want))), what

        h = px.builtin(f"scan:{dt}")
        keep = x > (0.5 if dt[0] == "f" else 0)
        hc = px.builtin(f"copy_if:{dt}:gt:{'0.5' if dt[0] == 'f' else '0'}")
        for a, b in ((0, 0), (es, es), (es, 0), (0, 3 * es)):  # input and output phases
            src, dst = dev(x.nbytes, a), dev(x.nbytes, b)
            put(src, x)
            torch.cuda.synchronize()
            assert lib.parallax_segmented_inclusive_scan(h, src[1], dst[1], n, o.data_ptr(), S) == px.OK
            close(get(dst), incl, ("inclusive", dt, a, b))
            assert lib.parallax_segmented_exclusive_scan(h, src[1], dst[1], n, o.data_ptr(), S,
                                                         init.ctypes.data) == px.OK
            close(get(dst), excl, ("exclusive", dt, a, b))
            counts = torch.full((S,), 77, dtype=torch.int64, device="cuda")
            dst[0].zero_()
            torch.cuda.synchronize()
            assert lib.parallax_segmented_copy_if(hc, src[1], dst[1], n, o.data_ptr(), S,
                                                  counts.data_ptr()) == px.OK
            got, k = get(dst), counts.cpu().numpy()
            for i, s in enumerate(seg):
                want = x[s][keep[s]]
                assert k[i] == want.size, (dt, i)
                assert np.array_equal(got[s][: want.size], want), (dt, i)
                assert not got[s][want.size:].any(), (dt, i)  # nothing beyond the kept ones
            assert lib.parallax_segmented_inclusive_scan(h, src[1], src[1], n, o.data_ptr(), S) == px.OK
            close(get(src), incl, ("in place", dt, a))
    print("segmented pipelines ok")


def test_pipelines_for_every_length(tmp_path):
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"{op} {t} {b} 1024 7\n" for op in (8, 16) for t in range(6)
                             for b in range(31)))
    r = subprocess.run([sys.executable, __file__], env=dict(os.environ, PARALLAX_TUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "segmented pipelines ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


if __name__ == "__main__":
    run_checks()
