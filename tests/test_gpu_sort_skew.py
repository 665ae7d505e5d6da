"""The tuple sort by units where one k-mer holds much of the input or few k-mers hold all of it: the oversized buckets beside
the units (spread over many blocks) or, where most tuples are in such buckets, the digit passes; against a stable host sort, and
that a skewed sort takes no more than a few times what an even one of its size does.
"""
import numpy as np
import pytest

from metapart_gb300 import native

pytestmark = pytest.mark.gpu


def _keys(n, share, seed, few=0):
    """share: of the tuples that one k-mer holds; few: the number of other k-mers (0: as many as tuples)."""
    rng = np.random.default_rng(seed)
    kmer = rng.integers(0, 1 << 62, size=n, dtype=np.uint64)
    if few:
        kmer = kmer[rng.integers(0, few, size=n)]
    kmer[rng.random(n) < share] = kmer[0]
    lo = (kmer << np.uint64(8)) | rng.integers(0, 64, size=n, dtype=np.uint64)
    return lo, (kmer >> np.uint64(56)).astype(np.uint8), np.arange(n, dtype=np.uint32)


def _sort(ctx, d, o):
    import torch
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    torch.cuda.synchronize()
    e[0].record()
    native.sort_tuples(ctx, *(x.data_ptr() for x in d + o), d[0].numel(), torch.cuda.current_stream().cuda_stream)
    e[1].record()
    torch.cuda.synchronize()
    return e[0].elapsed_time(e[1])


def _dev(lo, hi, ids):
    import torch
    return [torch.from_numpy(lo.view(np.int64)).cuda(), torch.from_numpy(hi).cuda(), torch.from_numpy(ids.view(np.int32)).cuda()]


# units beside one oversized bucket and beside several, the sample's lines (a bucket of a large block, half of the tuples,
# many tuples or few), digit passes for all
@pytest.mark.parametrize("n,share,few", [(3_000_000, 0.3, 0), (3_000_000, 0.45, 0), (3_000_000, 0.55, 0), (2_000_000, 0.007, 0),
                                         (2_500_000, 0.2, 400), (2_500_000, 0.0, 150), (1_572_863, 0.1, 0), (1_572_864, 0.1, 0),
                                         (60_000, 0.19, 0), (60_000, 0.3, 0), (12_500, 0.999, 0)])
def test_matches_stable_host_sort(built_gpu, n, share, few):
    import torch
    lo, hi, ids = _keys(n, share, n, few)
    order = np.lexsort((lo, hi))
    d = _dev(lo, hi, ids)
    o = [torch.empty_like(x) for x in d]
    with native.Context(0) as ctx:
        _sort(ctx, d, o)
    assert np.array_equal(o[2].cpu().numpy().view(np.uint32), ids[order])
    assert np.array_equal(o[0].cpu().numpy().view(np.uint64), lo[order])
    assert np.array_equal(o[1].cpu().numpy(), hi[order])


@pytest.mark.parametrize("share", [0.3, 0.9])
def test_one_kmer_is_not_one_block_s(built_gpu, share):
    import torch
    n = 4_000_000
    with native.Context(0) as ctx:
        t = []
        for s in (0.0, share):
            d = _dev(*_keys(n, s, 5))
            o = [torch.empty_like(x) for x in d]
            t.append(min(_sort(ctx, d, o) for _ in range(6)))
    assert t[1] < 6 * t[0], t


@pytest.mark.parametrize("n,share", [(2_000, 0.0), (40_000, 0.0), (3_000_000, 0.4)])
def test_budget_of_the_digit_passes_is_enough(built_gpu, n, share):
    """The smallest budget that the sort in place fits (digit passes alone), to a few KB, is enough for the other."""
    lo, hi, ids = _keys(n, share, 7)
    order = np.lexsort((lo, hi))

    def sort(budget, in_place):
        import torch
        d = _dev(lo, hi, ids)
        o = d if in_place else [torch.empty_like(x) for x in d]
        with native.Context(0, hbm_budget=budget) as ctx:
            try:
                _sort(ctx, d, o)
            except native.MetapartError as e:
                assert "(-4)" in str(e)  # MP_ENOMEM
                return None
        return o[2].cpu().numpy().view(np.uint32)

    small, fits = 1024, 256 << 20
    while fits - small > 4096:
        m = (small + fits) // 2
        if sort(m, True) is None:
            small = m
        else:
            fits = m
    for more in (0, 64 << 10, 1 << 20, 3 << 20, 5 << 20, 20 << 20, 40 << 20):
        got = sort(fits + more, False)
        assert got is not None and np.array_equal(got, ids[order]), (fits, more)
