"""A segmented call whose work list outgrows the segment buffer: the launch epoch starts again in the new
buffer, while the look-back entries of earlier calls lie in a buffer of their own that had room. They must not
read as the new call's. Sizes: 17,003 and then 19,503 possible work items, 56 bytes each against a 1 MiB buffer,
and 128 bytes each against a 4 MiB one. Integer prefixes, bit for bit; a thread of its own has fresh buffers."""
from __future__ import annotations

import threading

import pytest

pytestmark = pytest.mark.gpu

MIN_TILE = 256 * 3 * 4 - 4  # elements of the smallest tile


def test_epoch_restart_sees_no_old_entries(lib, px, dev, monkeypatch):
    monkeypatch.setenv("PARALLAX_TUNE", "0")
    torch = dev.torch
    bad = []

    def work():
        for seed, items in ((1, 17000), (2, 19500)):
            n = items * MIN_TILE
            gen = torch.Generator(device="cuda").manual_seed(seed)
            x = torch.randint(-1000, 1001, (n,), dtype=torch.int32, device="cuda", generator=gen)
            out = torch.zeros_like(x)
            off = torch.tensor([0, 5, n], dtype=torch.int64, device="cuda")
            want = torch.cat([torch.cumsum(x[:5], 0, dtype=torch.int32),
                              torch.cumsum(x[5:], 0, dtype=torch.int32)])
            torch.cuda.synchronize()
            st = lib.parallax_segmented_inclusive_scan(px.builtin("scan:i32"), x.data_ptr(), out.data_ptr(), n,
                                                       off.data_ptr(), 2)
            if st != px.OK or not torch.equal(out, want):
                bad.append((items, st, int((out != want).sum())))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not bad, bad
