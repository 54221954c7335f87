"""Segmented calls on whole-heap-capture memory: the operands lie in the page-locked host mirror and are used
in place, so they are read with plain loads, never bulk-copied: the tuner must not offer the pipelines, and
an untuned long-segment reduce must not take one. Results against numpy, in a process of its own (the heap
pool has to be live before the runtime's arena), with and without timing the candidates."""
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
    lens = np.array([50000, 0, 1, 70001, 3, 60000, 40003, 16384] * 4)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    n, S = int(off[-1]), len(lens)
    x = np.random.default_rng(3).integers(-1000, 1001, n).astype(np.int32)

    def pool(nbytes):
        p = raw.px_pool_alloc(nbytes, 256)
        assert p and raw.px_pool_contains(C.c_void_p(p))
        return p, np.ctypeslib.as_array((C.c_ubyte * nbytes).from_address(p)).view(np.int32)

    src, a = pool(x.nbytes)
    dst, out = pool(x.nbytes)
    a[:] = x
    o = torch.from_numpy(off.view(np.int64)).cuda()
    res = torch.zeros(S, dtype=torch.int32, device="cuda")
    counts = torch.zeros(S, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    seg = [slice(int(off[s]), int(off[s + 1])) for s in range(S)]
    assert lib.parallax_segmented_reduce(px.builtin("reduce:sum:i32"), src, n, o.data_ptr(), S,
                                         res.data_ptr()) == px.OK
    assert res.cpu().tolist() == [int(x[s].sum()) for s in seg]
    assert lib.parallax_segmented_inclusive_scan(px.builtin("scan:i32"), src, dst, n, o.data_ptr(), S) == px.OK
    assert np.array_equal(out, np.concatenate([np.cumsum(x[s], dtype=np.int32) for s in seg]))
    assert lib.parallax_segmented_copy_if(px.builtin("copy_if:i32:gt:0"), src, dst, n, o.data_ptr(), S,
                                          counts.data_ptr()) == px.OK
    for s, k in zip(seg, counts.cpu().tolist()):
        want = x[s][x[s] > 0]
        assert k == want.size and np.array_equal(out[s][:k], want)
    print("heap operands ok")


@pytest.mark.parametrize("tune", ["1", "0"])
def test_mirror_operands_take_plain_loads(tune):
    env = dict(os.environ, PARALLAX_DEBUG="1", PARALLAX_TUNE=tune, PARALLAX_HEAP_POOL="256")
    env.pop("PARALLAX_TUNE_CACHE", None)
    r = subprocess.run([sys.executable, __file__], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "heap operands ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
    lines = [ln for ln in r.stderr.splitlines() if "[parallax] segmented op" in ln]
    assert len(lines) == (9 if tune == "1" else 0), lines  # three candidates for each of the three calls
    assert not any("pipeline" in ln or "1024 threads" in ln for ln in lines), lines


if __name__ == "__main__":
    run_checks()
