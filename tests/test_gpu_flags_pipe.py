"""Compaction by a registered flags image on arrays that take the pipeline (more than a wave of 114688-byte
tiles): the first such sizes, an exactly full last tile, and sizes near a power of two, where the flags fill
their buffer. Moved values, compared bit for bit with the same selection made by torch."""
from __future__ import annotations

import pytest

from test_gpu_user_images import COPY_IF, PARTITION, funnel_handles

pytestmark = pytest.mark.gpu

WAVE = 2 * 148 * 114688
PIPE = 53760


def sizes(es):
    wave, pipe = WAVE // es, PIPE // es
    return [wave + 1, (wave // pipe + 2) * pipe, (1 << 27) - 4096, 1 << 27]


@pytest.mark.parametrize("dt", ["i32", "i64"])
def test_registered_flags_above_a_wave(lib, px, dev, dt):
    torch = dev.torch
    es, ty = (4, torch.int32) if dt == "i32" else (8, torch.int64)
    gen = torch.Generator(device="cuda").manual_seed(31)
    for n in sizes(es):
        x = torch.randint(-(1 << 30), 1 << 30, (n,), dtype=ty, device="cuda", generator=gen)
        keep = x % 3 == 0 if dt == "i32" else x & 1 != 0
        out = torch.empty_like(x)
        torch.cuda.synchronize()
        hs = (funnel_handles(lib, COPY_IF, "T = int; Pred = Mod3", "flags_mod3_i32") if dt == "i32"
              else funnel_handles(lib, COPY_IF, "T = long int; Pred = Odd", "flags_odd_i64"))
        k = lib.parallax_copy_if(*hs, x.data_ptr(), out.data_ptr(), n, es, 0)
        px.check("copy_if")
        want = x[keep]
        assert k == want.numel() and torch.equal(out[:k], want), n
        if dt == "i32":
            keep = x < 0
            hs = funnel_handles(lib, PARTITION, "T = int; Pred = Neg", "flags_neg_i32")
        else:
            hs = funnel_handles(lib, PARTITION, "T = long int; Pred = Odd", "flags_odd_i64")
        k = lib.parallax_copy_if(*hs, x.data_ptr(), out.data_ptr(), n, es, 0)
        px.check("partition")
        want = torch.cat([x[keep], x[~keep]])
        assert k == int(keep.sum()) and torch.equal(out, want), n
        del x, keep, out, want
