"""Calls captured into a CUDA graph after a warm-up with small arrays only: no workspace buffer may have to grow
for the look-back entries of a 480 MB scan or selection, for 9,800 work items of a segmented call, or for a sort
of 2^18 keys. Each graph is launched once; results against torch. A thread of its own has fresh buffers."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_capture_after_a_small_warm_up(lib, px, dev, monkeypatch):
    monkeypatch.setenv("PARALLAX_TUNE", "0")
    torch = dev.torch
    n, m, k = 120_000_000, 30_000_000, 1 << 18
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(-1000, 1001, (n,), dtype=torch.int32, device="cuda", generator=gen)
    y = torch.zeros_like(x)
    off = torch.tensor([0, 7, m], dtype=torch.int64, device="cuda")
    few = torch.tensor([0, 7, 1000], dtype=torch.int64, device="cuda")
    keys = torch.randint(-(1 << 31), 1 << 31, (k,), dtype=torch.int64, device="cuda",
                         generator=gen).to(torch.int32)
    zero = np.zeros(1, np.int32)
    hs, hc, hk = px.builtin("scan:i32"), px.builtin("copy_if:i32:gt:0"), px.builtin("sort:i32")
    calls = {
        "scan": lambda small: lib.parallax_exclusive_scan(hs, hs, hs, x.data_ptr(), y.data_ptr(),
                                                          1000 if small else n, 4, zero.ctypes.data),
        "copy_if": lambda small: lib.parallax_copy_if(hc, hc, hc, hc, x.data_ptr(), y.data_ptr(),
                                                      1000 if small else n, 4, 0),
        "segmented": lambda small: lib.parallax_segmented_inclusive_scan(
            hs, x.data_ptr(), y.data_ptr(), 1000 if small else m, (few if small else off).data_ptr(), 2),
        "sort": lambda small: lib.parallax_sort(hk, keys.data_ptr(), 100_000 if small else k, 4),
    }
    problems = []

    def work():
        for name, call in calls.items():
            s = torch.cuda.Stream()
            torch.cuda.synchronize()
            lib.parallax_set_stream(s.cuda_stream)
            lib.parallax_set_async(1)
            call(True)
            lib.parallax_synchronize()
            want = {"scan": lambda: torch.cumsum(x, 0, dtype=torch.int32) - x, "copy_if": lambda: x[x > 0],
                    "segmented": lambda: torch.cat([torch.cumsum(x[:7], 0, dtype=torch.int32),
                                                    torch.cumsum(x[7:m], 0, dtype=torch.int32)]),
                    "sort": lambda: torch.sort(keys).values}[name]()
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            try:
                with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
                    lib.parallax_clear_error()
                    call(False)
                    status = lib.parallax_last_error()
                if status != px.OK:
                    problems.append((name, status))
                else:
                    g.replay()
                    torch.cuda.synchronize()
                    got = (keys if name == "sort" else y)[:want.numel()]
                    if not torch.equal(got, want):
                        problems.append((name, "differs"))
            except RuntimeError as e:
                problems.append((name, str(e)[:100]))
            lib.parallax_clear_error()
            lib.parallax_set_async(0)
            lib.parallax_set_stream(None)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not problems, problems
