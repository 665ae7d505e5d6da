"""The tuple sort by units (k_unit_rank) against a stable host sort by the whole 72-bit key: sizes at its lower end, key
widths from one byte above the window to nine bytes, and the tuples that leave its common path -- bins of equal keys
above the comparison limit, buckets above one block's and two blocks' capacity, constant bits above the window, and
a sort in place."""
import numpy as np
import pytest

from metapart_gb300 import native

pytestmark = pytest.mark.gpu

N0 = 1 << 10
CASES = [(n, 70, "even") for n in (N0 - 1, N0, N0 + 1)] + [(1_000_003, b, "even") for b in (72, 70, 66, 64, 62, 50, 38, 25)] + [
    (700_001, 70, "copies"), (700_001, 62, "copies"), (900_007, 70, "mid"), (900_007, 62, "mid"), (900_007, 70, "big"),
    (600_000, 62, "big"), (400_001, 70, "high bits"), (400_001, 38, "high bits"), (400_001, 72, "narrow"), (300_000, 70, "in place")]


def _keys(n, bits, kind, rng):
    lo = rng.integers(0, 1 << 64, size=n, dtype=np.uint64)
    hi = rng.integers(0, 256, size=n, dtype=np.uint64)
    if bits < 64:
        lo &= np.uint64((1 << bits) - 1)
    hi &= np.uint64((1 << max(0, bits - 64)) - 1)
    if kind == "copies":    # a few hundred keys of 2,000 copies beside keys of their own
        m = rng.integers(0, 300, size=n)
        few = rng.random(n) < 0.8
        lo, hi = np.where(few, lo[m], lo), np.where(few, hi[m], hi)
    if kind in ("mid", "big"):  # buckets of 9,000 and 60,000 tuples that differ in their low bits only
        each = 9_000 if kind == "mid" else 60_000
        m = np.arange(n) // each
        few = m < (n // each) // 2
        low = np.uint64((1 << 40) - 1)
        lo, hi = np.where(few, (lo[m] & ~low) | (lo & low), lo), np.where(few, hi[m], hi)
        p = rng.permutation(n)
        lo, hi = lo[p], hi[p]
    if kind == "high bits":
        lo |= np.uint64(1 << 63)
    if kind == "narrow":    # the varying bits start below the word's top
        lo = (lo & np.uint64((1 << 45) - 1)) | np.uint64(0x5A << 56)
        hi[:] = 0x3C
    return lo, hi


@pytest.mark.parametrize("n,bits,kind", CASES, ids=[f"{c[2]}-{c[0]}-{c[1]}" for c in CASES])
def test_unit_sort_matches_stable_host_sort(built_gpu, n, bits, kind):
    import torch
    rng = np.random.default_rng(n + bits)
    lo, hi = _keys(n, bits, kind, rng)
    ids = rng.integers(0, 1 << 32, size=n, dtype=np.uint32)
    has_hi = bits > 64
    order = np.lexsort((lo, hi)) if has_hi else np.argsort(lo, kind="stable")
    d = [torch.from_numpy(lo.view(np.int64)).cuda(), torch.from_numpy(hi.astype(np.uint8)).cuda() if has_hi else None,
         torch.from_numpy(ids.view(np.int32)).cuda()]
    o = d if kind == "in place" else [None if x is None else torch.empty_like(x) for x in d]
    p = [None if x is None else x.data_ptr() for x in d + o]
    with native.Context(0) as ctx:
        native.sort_tuples(ctx, *p, n)
    assert np.array_equal(o[0].cpu().numpy().view(np.uint64), lo[order])
    assert np.array_equal(o[2].cpu().numpy().view(np.uint32), ids[order])
    if has_hi:
        assert np.array_equal(o[1].cpu().numpy(), hi.astype(np.uint8)[order])
    if kind != "in place":
        assert np.array_equal(d[0].cpu().numpy().view(np.uint64), lo)  # the input stays
