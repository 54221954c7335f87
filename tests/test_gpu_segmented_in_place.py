"""Segmented selections written over their input: the first call of a kind must not time its candidates there,
since every timed run would compact what the one before has left. Types and operations are ones that no other
test has timed for the length (mean 2^21); several calls in a row."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["copy_if", "remove_if", "unique"])
@pytest.mark.parametrize("dt", ["u32", "u64"])
def test_selection_over_its_input(lib, px, dev, op, dt):
    torch = dev.torch
    ty = torch.int32 if dt == "u32" else torch.int64
    S, length = 3, 1 << 21
    n = S * length
    off = torch.arange(S + 1, dtype=torch.int64, device="cuda") * length
    counts = torch.zeros(S, dtype=torch.int64, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(12)
    for _ in range(2):
        x = torch.randint(0, 4, (n,), device="cuda", generator=gen).to(ty)
        if op == "unique":
            keep = torch.ones(n, dtype=torch.bool, device="cuda")
            keep[1:] = x[1:] != x[:-1]
            keep[off[:-1]] = True
            h, fn = px.builtin(f"unique:{dt}"), lib.parallax_segmented_unique
        else:
            keep = (x > 1) == (op == "copy_if")
            h, fn = px.builtin(f"{op}:{dt}:gt:1"), lib.parallax_segmented_copy_if
        want = [x[s * length:(s + 1) * length][keep[s * length:(s + 1) * length]] for s in range(S)]
        torch.cuda.synchronize()
        assert fn(h, x.data_ptr(), x.data_ptr(), n, off.data_ptr(), S, counts.data_ptr()) == px.OK
        assert counts.cpu().tolist() == [w.numel() for w in want]
        for s, w in enumerate(want):
            assert torch.equal(x[s * length:s * length + w.numel()], w), s
