"""The tuner keeps apart the calls that a pipeline takes and those it does not: operands in HBM and in the
page-locked host mirror (whole-heap capture) of one mean length, in turn, time their candidates once, and the
choice for one is not forced on the other. Files of either kind of entry are used without timing. In processes
of their own, because the tuner reads its file once."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
S, LENGTH = 64, 300_000  # bucket 18


def run_checks() -> None:
    import torch

    sys.path.insert(0, str(ROOT))
    import __graft_entry__ as g

    px = g._pkg()
    raw = C.CDLL(str(px.LIB_PATH))
    raw.px_pool_alloc.restype = C.c_void_p
    raw.px_pool_alloc.argtypes = [C.c_size_t, C.c_size_t]
    assert raw.px_pool_init() == 1
    lib = px.load()
    assert lib.parallax_arena_alloc(64, 64)  # starts the arena, which adopts the pool
    n = S * LENGTH
    x = np.random.default_rng(3).integers(-1000, 1001, n).astype(np.int32)
    dx = torch.from_numpy(x).cuda()
    dy = torch.zeros_like(dx)
    p, q = raw.px_pool_alloc(x.nbytes, 256), raw.px_pool_alloc(x.nbytes, 256)
    np.ctypeslib.as_array((C.c_ubyte * x.nbytes).from_address(p)).view(np.int32)[:] = x
    out = np.ctypeslib.as_array((C.c_ubyte * x.nbytes).from_address(q)).view(np.int32)
    o = torch.arange(S + 1, dtype=torch.int64, device="cuda") * LENGTH
    r = torch.zeros(S, dtype=torch.int32, device="cuda")
    sums = x.reshape(S, LENGTH).sum(axis=1, dtype=np.int32)
    scans = np.cumsum(x.reshape(S, LENGTH), axis=1, dtype=np.int32).ravel()
    torch.cuda.synchronize()
    for src, dst in ((dx.data_ptr(), dy.data_ptr()), (p, q)) * 2:
        assert lib.parallax_segmented_reduce(px.builtin("reduce:sum:i32"), src, n, o.data_ptr(), S,
                                             r.data_ptr()) == px.OK
        assert np.array_equal(r.cpu().numpy(), sums)
        r.zero_()
        torch.cuda.synchronize()
        assert lib.parallax_segmented_inclusive_scan(px.builtin("scan:i32"), src, dst, n, o.data_ptr(),
                                                     S) == px.OK
    assert np.array_equal(dy.cpu().numpy(), scans) and np.array_equal(out, scans)
    print("tuner ok")


def run(cache) -> list[str]:
    env = dict(os.environ, PARALLAX_DEBUG="1", PARALLAX_HEAP_POOL="512", PARALLAX_TUNE_CACHE=str(cache))
    env.pop("PARALLAX_TUNE", None)
    r = subprocess.run([sys.executable, __file__], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "tuner ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
    return [ln for ln in r.stderr.splitlines() if "tuned segmented op" in ln]


def test_pipelines_have_their_own_entries(tmp_path):
    cache = tmp_path / "tune.txt"
    tuned = run(cache)
    assert len(tuned) == 2, tuned  # reduce and scan, once each, though four calls of each ran
    e = {tuple(ln.split()[:3]): ln.split()[3:] for ln in cache.read_text().splitlines()}
    assert set(e) == {(op, "2", "18") for op in ("0", "64", "8", "72")}, e
    assert e["72", "2", "18"] == ["1024", "7"] and e["8", "2", "18"] != ["1024", "7"], e
    assert e["64", "2", "18"] == ["512", "7"] and e["0", "2", "18"] != ["512", "7"], e
    assert run(cache) == []  # and the file is enough


def test_files_without_pipeline_entries(tmp_path):
    cache = tmp_path / "tune.txt"
    cache.write_text("0 2 18 256 7\n8 2 18 256 7\n")
    assert run(cache) == []  # used as they are
    cache.write_text("0 2 18 512 7\n8 2 18 1024 7\n")
    tuned = run(cache)  # a pipeline's shape says nothing for operands it does not take
    assert len(tuned) == 1 and "op 8" in tuned[0], tuned


if __name__ == "__main__":
    run_checks()
