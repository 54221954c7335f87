"""Padding of the flags array that a registered predicate image writes: the compaction kernels read the
flags of whole tiles, so the array has to reach to the end of the last tile of every kernel's shape.
Checked on the CPU, over the header that the kernels take their shapes from."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "parallax-runtime_b200" / "csrc"

PROGRAM = r"""
#include "compact_shape.hpp"
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
int main(int argc, char** argv) {
    for (int i = 1; i < argc; ++i) {
        const size_t n = strtoull(argv[i], nullptr, 10);
        size_t end = 0;
        for (size_t elem : {size_t(4), size_t(8)})
            for (size_t tile : {pxb::compact_tile(elem), pxb::compact_pipe_tile(elem)}) {
                const size_t e = (n + tile - 1) / tile * tile;
                if (e > end) end = e;
            }
        printf("%zu %zu\n", end, pxb::compact_flags_padding(n));
    }
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "shape.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(d / "shape.cpp"), "-o",
                    str(d / "shape")], check=True)

    def go(ns):
        out = subprocess.run([str(d / "shape"), *map(str, ns)], capture_output=True, text=True, check=True)
        return [tuple(map(int, ln.split())) for ln in out.stdout.splitlines()]
    return go


def test_flags_reach_the_last_tile_of_every_shape(run):
    tiles = [28672, 14336, 13440, 6720]
    ns = [1, 2, 1000, (1 << 20) + 7, 4243457, 8486913, 134213632, 268420608, (1 << 32) + 5]
    ns += [k * t + d for t in tiles for k in (1, 2, 3, 297, 633, 4682, 19973) for d in (-1, 0, 1)]
    for n, (end, padded) in zip(ns, run(ns)):
        assert padded >= end >= n, (n, end, padded)
        assert padded <= n + max(tiles) + 16, (n, padded)  # and not more than it needs
