"""Rules of the kernels that a run cannot show, checked on the source text: a broken one gives wrong
results only when the timing is unlucky.

* Kernels launched as dependents (pdl.cuh) start while earlier kernels of their stream still write, so
  they and their device functions use no read-only load: no __ldg, ld.global.nc or __restrict__.
* In the pipelines one lane arrives for its warp on the barrier that lets other warps, and in the end the
  mover, write to a buffer and its slot. Between the wait that gave the warp the slot and the arrival the
  whole warp meets (__syncwarp, or a warp reduction that every lane takes part in), so that no lane still
  reads the slot.
* Every wait between warps ends by itself: they meet at an mbarrier, polled up to a limit (wait_bar), not
  at a named barrier, which waits forever for a warp that gave up another wait."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "parallax-runtime_b200" / "csrc"


def files() -> list[Path]:
    # csrc/lto holds modules that are linked at run time and launched plainly
    return sorted(f for e in ("*.cu", "*.cuh") for f in CSRC.rglob(e) if f.parent.name != "lto")


def functions(text: str) -> list[str]:
    """Device code in pieces that each begin at a __global__ or __device__ function."""
    text = re.sub(r"//[^\n]*", "", text)
    cuts = [m.start() for m in re.finditer(r"__global__|__device__ __forceinline__", text)]
    return [text[a:b] for a, b in zip(cuts, cuts[1:] + [len(text)])]


def test_dependent_kernels_use_no_read_only_loads():
    kernels = 0
    for f in files():
        for fn in functions(f.read_text()):
            plain = fn.startswith("__global__") and "dependent_prologue()" not in fn
            kernels += fn.startswith("__global__") and not plain
            bad = re.findall(r"\b__ldg\b|\bldg_stream16\b|ld\.global\.nc|__restrict__", fn)
            if bad and not plain and " ldg_stream16(const void* p) {" not in fn:
                raise AssertionError((f.name, bad, fn[:200]))
    assert kernels > 15  # the dependent kernels were found


def test_warps_meet_before_a_lane_arrives_for_them():
    arrivals = 0
    for f in files():
        for fn in functions(f.read_text()):
            if not fn.startswith("__global__"):
                continue
            for m in re.finditer(r"mbar_arrive\(&(\w+)\[", fn):
                if m.group(1) == "full":  # the mover, a single lane
                    continue
                arrivals += 1
                waits = [w.end() for w in re.finditer(r"\bwait_bar\(|\blanded\(", fn[:m.start()])]
                since = fn[waits[-1]:m.start()]
                assert "__syncwarp();" in since or "__reduce_add_sync(" in since, (f.name, m.group(0), since)
    assert arrivals >= 15


def test_no_unbounded_named_barriers():
    for f in files():
        assert not re.search(r"\bbar\.sync\b|\bbarrier\.sync\b|\bbarrier\.cta\.sync\b", f.read_text()), f.name
