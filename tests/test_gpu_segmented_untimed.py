"""Segmented calls that time no candidates (PARALLAX_TUNE=0, in-place scans) pick their kernel by the mean segment
length alone: every operation just below and at the lengths where the rule turns (2048, 8192, 16384), against
torch, integers bit for bit. In a process of its own, in which no other test has timed anything."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def run_checks() -> None:
    import torch

    sys.path.insert(0, str(ROOT))
    import __graft_entry__ as g

    px = g._pkg()
    lib = px.load()
    S = 40
    gen = torch.Generator(device="cuda").manual_seed(2)
    for dt, ty in (("i32", torch.int32), ("i64", torch.int64)):
        for mean in (2047, 2048, 8191, 8192, 16383, 16384):
            n = S * mean
            cuts = torch.randperm(n - 1, device="cuda", generator=gen)[: S - 1].sort().values + 1
            off = torch.cat([cuts.new_zeros(1), cuts, cuts.new_full((1,), n)])
            seg = list(zip(off[:-1].tolist(), off[1:].tolist()))
            x = torch.randint(-1000, 1001, (n,), device="cuda", generator=gen).to(ty)
            y, r = torch.zeros_like(x), torch.zeros(S, dtype=ty, device="cuda")
            counts = torch.zeros(S, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            o, c = off.data_ptr(), counts.data_ptr()
            assert lib.parallax_segmented_reduce(px.builtin(f"reduce:max:{dt}"), x.data_ptr(), n, o, S,
                                                 r.data_ptr()) == px.OK
            assert r.tolist() == [int(x[a:b].max()) for a, b in seg]
            z = x.clone()
            torch.cuda.synchronize()
            assert lib.parallax_segmented_inclusive_scan(px.builtin(f"scan:{dt}"), z.data_ptr(), z.data_ptr(), n,
                                                         o, S) == px.OK
            assert torch.equal(z, torch.cat([torch.cumsum(x[a:b], 0, dtype=ty) for a, b in seg])), (dt, mean)
            keep = x > 0
            for name, spec in (("copy_if", f"copy_if:{dt}:gt:0"), ("partition", f"partition:{dt}:gt:0"),
                               ("unique", f"unique:{dt}")):
                fn = getattr(lib, f"parallax_segmented_{name}")
                assert fn(px.builtin(spec), x.data_ptr(), y.data_ptr(), n, o, S, c) == px.OK
                for (a, b), k in zip(seg, counts.tolist()):
                    v, m = x[a:b], keep[a:b]
                    want = (v[m] if name == "copy_if" else torch.cat([v[m], v[~m]]) if name == "partition"
                            else torch.unique_consecutive(v))
                    assert k == (int(m.sum()) if name == "partition" else want.numel()), (name, dt, mean)
                    assert torch.equal(y[a:a + want.numel()], want), (name, dt, mean)
    print("untimed calls ok")


def test_rule_by_mean_length():
    env = dict(os.environ, PARALLAX_TUNE="0")
    env.pop("PARALLAX_TUNE_CACHE", None)
    r = subprocess.run([sys.executable, __file__], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "untimed calls ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


if __name__ == "__main__":
    run_checks()
