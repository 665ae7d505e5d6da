"""The grouped scan (k_group.cu) against the sorted one: a job whose scans are split into units and grouped by
k-mer gives the labels, bounds and partition files of the same job with its scans sorted (a job with the
self-checks on sorts them, and the parity tests pin that path to the oracle).

The inputs sit where the split and the tables change: one level and two, units at and above a block's capacity
(buckets of a 200 bp genome hold tens of thousands of tuples), runs that branch on one side or both, thread ranges
of one bucket, scans whose every k-mer occurs once, one k-mer in the whole input, and the sweeps' initial state
(a range whose first valid tuple carries the scan's last k-mer, with a first read that is BAD or not).
"""
import numpy as np
import pytest

from metapart_gb300 import native, synth
from test_gpu_batch import _poly_c
from test_oracle_bad_anchor import _mg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(built_gpu):
    c = native.Context(0)
    yield c
    c.close()


def _run(ctx, data, k, chunks, scans, threads, il, min3, store, sort):
    fno, ofs = native.fastq_index(chunks, [data], il)
    starts = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.set_checks(sort)
        job.set_read_store(store)
        job.load(data, interleaved=il)
        cnt = job.count(k, starts, min3)
        b = job.partition(k, scans, threads, starts, cnt.chunk_first_read, cnt.hist, min3)
        out, sizes = job.output()
        return b.copy(), job.labels(), sizes.copy(), np.array(out), job.sort_split()["unit_passes"]


def _same(ctx, data, k, chunks, scans, threads, il=False, min3=False, store="kmer_cache", grouped=True):
    a = _run(ctx, data, k, chunks, scans, threads, il, min3, store, False)
    b = _run(ctx, data, k, chunks, scans, threads, il, min3, store, True)
    assert not grouped or a[4] == 0  # no unit was sorted
    for x, y in zip(a[:4], b[:4]):
        assert np.array_equal(x, y)


CASES = [
    ("plain_large", 200_000, 31, 16, 1, 16, False, False, "kmer_cache"),   # two levels
    ("plain_large", 60_000, 31, 16, 2, 4, False, False, "packed"),
    ("plain_large", 9_000, 29, 8, 1, 8, False, False, "kmer_cache"),       # one level, most k-mers once
    ("plain_small", 30_000, 27, 16, 1, 16, False, False, "fastq"),
    ("plain_small", 20_000, 21, 8, 3, 2, False, False, "kmer_cache"),
    ("plain_small", 8_000, 11, 4, 2, 2, False, False, "kmer_cache"),
    ("interleaved_small", 30_000, 27, 16, 2, 2, True, False, "kmer_cache"),
    ("hotspot", 9_000, 31, 4, 1, 2, False, False, "kmer_cache"),           # buckets of a few thousand tuples
    ("hotspot", 40_000, 25, 12, 2, 3, False, False, "packed"),             # and above a unit's capacity
    ("min3", 20_000, 31, 16, 1, 4, False, True, "kmer_cache"),
    ("plain_small", 600, 27, 256, 1, 256, False, False, "kmer_cache"),     # thread ranges of a bucket or none
    ("hotspot", 300, 27, 64, 2, 64, False, False, "kmer_cache"),
]


@pytest.mark.parametrize("name,n,k,chunks,scans,threads,il,min3,store", CASES,
                         ids=[f"{c[0]}-{c[1]}-k{c[2]}-s{c[4]}-t{c[5]}" for c in CASES])
def test_grouped_equals_sorted(ctx, name, n, k, chunks, scans, threads, il, min3, store):
    _same(ctx, synth.fastq_bytes(synth.workload(name, n, seed=71)), k, chunks, scans, threads, il, min3, store)


@pytest.mark.parametrize("threads", [1, 2])
@pytest.mark.parametrize("variant", range(3))
def test_bad_first_read(ctx, variant, threads):
    mg = _mg()
    two = mg.BAD_ANCHOR[variant] == "two_scans"  # its second scan starts from a hooked BAD read and is sorted
    _same(ctx, mg.bad_anchor_fastq(variant), 27, 4, 2 if two else 1, threads, grouped=not two)


@pytest.mark.parametrize("threads", [1, 4])
def test_one_kmer(ctx, threads):
    _same(ctx, _poly_c(3000), 31, 4, 1, threads)  # one run of 210,000 tuples: the scan's last and its first


@pytest.mark.parametrize("seed", range(6))
def test_random_tiny(ctx, seed):
    """Two to forty reads cut from a 90 bp genome with some errors: most ranges hold one or two runs, so the sweeps'
    initial state acts in many of them."""
    rng = np.random.default_rng(seed)
    for _ in range(12):
        n, scans, threads = 2 * int(rng.integers(1, 20)), int(rng.integers(1, 3)), int(rng.integers(1, 5))
        g = rng.choice(list(b"ACGT"), 90).astype(np.uint8)
        recs = []
        for i in range(n):
            p = int(rng.integers(0, 50))
            s = g[p:p + 40].copy()
            err = rng.random(40) < 0.02
            s[err] = rng.choice(list(b"ACGT"), int(err.sum()))
            recs.append(b"@t%d\n" % i + s.tobytes() + b"\n+\n" + b"I" * 40 + b"\n")
        data = b"".join(recs)
        starts = np.array([0] + [len(data)] * threads, dtype=np.uint64)
        starts = np.sort(np.r_[starts[:1], np.cumsum([len(r) for r in recs])[np.linspace(0, n - 1, threads).astype(int)]]).astype(np.uint64)
        starts[-1] = len(data)
        res = []
        for sort in (False, True):
            with native.Job(ctx) as job:
                job.set_checks(sort)
                job.load(data)
                cnt = job.count(21, starts)
                try:
                    b = job.partition(21, scans, threads, starts, cnt.chunk_first_read, cnt.hist)
                    res.append((b.tolist(), job.labels().tolist()))
                except native.MetapartError as e:  # ranges the planner refuses are refused on both paths
                    res.append(str(e))
        assert res[0] == res[1]


@pytest.mark.parametrize("k", [11, 17, 21, 31])
@pytest.mark.parametrize("scans", [2, 3])
@pytest.mark.parametrize("n", [600, 60_000])
def test_scans_split_together(ctx, n, scans, k):
    """Two and three scans whose first split pass is one, against a pass per scan (a piece limit that all scans
    together exceed): bins of every width, small scans' and (60,000 reads) the 1024-bucket bins that the scans' bounds cut."""
    data = synth.fastq_bytes(synth.workload("plain_large", n, seed=5 + k))
    fno, ofs = native.fastq_index(4, [data], False)
    starts = native.chunk_starts_of(fno, ofs, [len(data)])
    res = []
    for cap in (0, 1):
        with native.Job(ctx) as job:
            job.load(data)
            cnt = job.count(k, starts)
            total = int(cnt.hist[-1])
            if cap:
                job.set_scan_piece_tuples(total - 1)  # more than a scan, less than all
            b = job.partition(k, scans, 4, starts, cnt.chunk_first_read, cnt.hist)
            assert job.scan_pieces == scans
            out, sizes = job.output()
            res.append((b.tolist(), job.labels().tolist(), sizes.tolist(), bytes(out)))
    assert res[0] == res[1]
