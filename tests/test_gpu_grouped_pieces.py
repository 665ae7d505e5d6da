"""Scans in bucket-range pieces, grouped: against sorted pieces (a job with the self-checks runs both and compares parents, BAD
flags and hooked reads) and against whole scans.  The pieces cut thread ranges anywhere, hold one bucket or many, end or do not
end a range, and the sweeps' initial state (the scan's last run and first read) spans them.
"""
import time

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


def _run(ctx, data, starts, k, scans, threads, cap, checks=False):
    with native.Job(ctx) as job:
        job.set_checks(checks)
        job.set_scan_piece_tuples(cap)
        job.load(data)
        cnt = job.count(k, starts)
        b = job.partition(k, scans, threads, starts, cnt.chunk_first_read, cnt.hist)
        return b.tolist(), job.labels().tolist(), job.scan_pieces, job.sort_split()["unit_passes"], int(cnt.hist[-1])


def _compare(ctx, data, starts, k, scans, threads, caps):
    whole = _run(ctx, data, starts, k, scans, threads, 0)
    for cap in caps:
        got = _run(ctx, data, starts, k, scans, threads, cap)
        assert got[3] == 0  # no unit was sorted
        assert got[:2] == whole[:2], cap
        checked = _run(ctx, data, starts, k, scans, threads, cap, True)
        assert checked[:3] == got[:3], cap


def _starts(data, chunks):
    fno, ofs = native.fastq_index(chunks, [data])
    return native.chunk_starts_of(fno, ofs, [len(data)])


@pytest.mark.parametrize("name,n,k,scans,threads,caps", [
    ("plain_large", 40_000, 31, 2, 4, (400_000, 2_000_000)), ("plain_small", 20_000, 21, 3, 2, (60_000,)),
    ("plain_small", 8_000, 11, 1, 8, (50_000,)), ("hotspot", 30_000, 25, 1, 2, (20_000, 150_000)),
    ("hotspot", 30_000, 27, 2, 8, (90_000,)), ("plain_small", 600, 27, 1, 256, (2_000,))],
    ids=["large-s2", "small-s3", "k11", "hotspot", "hotspot-s2", "600-t256"])
def test_pieces(ctx, name, n, k, scans, threads, caps):
    data = synth.fastq_bytes(synth.workload(name, n, seed=61))
    _compare(ctx, data, _starts(data, 256 if threads == 256 else 16), k, scans, threads, caps)


@pytest.mark.parametrize("threads", [1, 4])
def test_one_kmer(ctx, threads):
    data = _poly_c(3000) + synth.fastq_bytes(synth.workload("plain_small", 400, seed=2))
    _compare(ctx, data, _starts(data, 4), 31, 1, threads, (5_000, 100_000))


@pytest.mark.parametrize("threads", [1, 2])
@pytest.mark.parametrize("variant", range(2))
def test_bad_first_read(ctx, variant, threads):
    data = _mg().bad_anchor_fastq(variant)
    st = _starts(data, 4)
    for cap in (296, 300):
        got = _run(ctx, data, st, 27, 1, threads, cap)
        assert got[2] > 1 and got[:3] == _run(ctx, data, st, 27, 1, threads, cap, True)[:3]
        assert got[:2] == _run(ctx, data, st, 27, 1, threads, 0)[:2]


@pytest.mark.parametrize("seed", range(6))
def test_random_tiny(ctx, seed):
    """Two to forty reads cut from a 90 bp genome with some errors: most ranges and pieces hold one or two runs."""
    rng = np.random.default_rng(100 + seed)
    for _ in range(8):
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
        ends = np.cumsum([len(r) for r in recs])[np.linspace(0, n - 1, threads).astype(int)]
        starts = np.sort(np.r_[0, ends]).astype(np.uint64)
        starts[-1] = len(data)
        cap = int(rng.integers(1, 20 * n // 2 + 2))
        res = []
        for c, checks in ((0, False), (cap, False), (cap, True)):
            try:
                res.append(_run(ctx, data, starts, 21, scans, threads, c, checks)[:2])
            except native.MetapartError as e:  # ranges the planner refuses are refused by all
                assert "check" not in str(e)
                res.append(str(e))
        assert res[0] == res[1] == res[2]


def test_time(ctx):
    """Sixteen pieces a scan take no more than so many times the whole scans: each makes two passes over the reads."""
    data = synth.fastq_bytes(synth.workload("plain_large", 1_000_000, seed=1))
    st = _starts(data, 16)
    t = {}
    with native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(31, st)
        for cap in (0, 8_000_000):
            job.set_scan_piece_tuples(cap)
            best = 1e9
            for _ in range(4):
                t0 = time.perf_counter()
                job.partition(31, 2, 16, st, cnt.chunk_first_read, cnt.hist)
                best = min(best, time.perf_counter() - t0)
            t[cap] = best * 1e3
        assert job.scan_pieces == 16
    assert t[8_000_000] < 11 * t[0], t
