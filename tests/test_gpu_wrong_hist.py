"""A histogram that is not the reads' (the FASTQ changed between the counting and the partitioning process, another k,
a damaged file): refused with MP_EFMT, by the split passes' own counts, and the job then partitions with the right one.
"""
import numpy as np
import pytest

from metapart_gb300 import native, synth
from test_gpu_batch import _poly_c
from test_gpu_errors import EFMT, code

pytestmark = pytest.mark.gpu

EUNSUP = -5


@pytest.fixture(scope="module")
def ctx(built_gpu):
    c = native.Context(0)
    yield c
    c.close()


def _moved(c, a, b, n=1):
    c[a] -= n
    c[b] += n


def _far(c):
    p = np.flatnonzero(c)
    _moved(c, p[0], p[-1])


def _far_back(c):
    p = np.flatnonzero(c)
    _moved(c, p[-1], p[0])


def _near(c):  # two units on
    p = np.flatnonzero(c)
    _moved(c, p[len(p) // 3], np.searchsorted(np.cumsum(c), c[:p[len(p) // 3]].sum() + 13_000))


def _emptied(c):  # tuples arrive where the histogram has none (many reads: in a whole bin)
    p = np.flatnonzero(c)
    lo, hi = (512 << 10, 513 << 10) if c.sum() > 2_000_000 else (p[4 * len(p) // 10], p[6 * len(p) // 10])
    n = c[lo:hi].sum()
    c[lo:hi] = 0
    c[np.flatnonzero(c)[0]] += n


def _more(c):
    c[np.flatnonzero(c)[-1]] += 7


def _less(c):  # (not the last bucket's, which the scans then end before)
    p = np.flatnonzero(c)
    c[p[len(p) // 2]] -= 1


def _halved(c):
    c //= 2


def _thrown(c):  # every count moved on by 1,000 buckets: the last tuples run past all places
    c[:] = np.roll(c, 1000)


WRONG = [_far, _far_back, _near, _emptied, _more, _less, _halved, _thrown]


@pytest.mark.parametrize("wrong", WRONG, ids=[f.__name__ for f in WRONG])
@pytest.mark.parametrize("name,n,k,scans,min3", [("plain_small", 600, 27, 1, False), ("plain_small", 600, 21, 2, False),
                                                 ("plain_large", 60_000, 31, 1, False), ("plain_large", 60_000, 31, 2, False),
                                                 ("plain_large", 60_000, 29, 3, False), ("min3", 40_000, 31, 1, True)],
                         ids=["600", "600-s2", "60000", "60000-s2", "60000-s3", "min3"])
def test_refused(ctx, name, n, k, scans, min3, wrong):
    data = synth.fastq_bytes(synth.workload(name, n, seed=19))
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(k, st, min3)
        want = job.partition(k, scans, 4, st, cnt.chunk_first_read, cnt.hist, min3), job.labels()
        c = np.diff(cnt.hist.astype(np.int64))
        wrong(c)
        assert (c >= 0).all()
        bad = np.r_[0, np.cumsum(c)].astype(np.uint64)
        with pytest.raises(native.MetapartError) as e:
            job.partition(k, scans, 4, st, cnt.chunk_first_read, bad, min3)
        assert code(e.value) == EFMT
        got = job.partition(k, scans, 4, st, cnt.chunk_first_read, cnt.hist, min3), job.labels()
        for a, b in zip(want, got):
            assert np.array_equal(a, b)


def test_histogram_of_another_k(ctx):
    data = synth.fastq_bytes(synth.workload("plain_large", 20_000, seed=20))
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.load(data)
        for k, other in ((31, 29), (29, 31)):
            cnt = job.count(other, st)
            for scans in (1, 2):
                with pytest.raises(native.MetapartError) as e:
                    job.partition(k, scans, 4, st, cnt.chunk_first_read, cnt.hist)
                assert code(e.value) == EFMT


@pytest.mark.parametrize("threads", [1, 2])
@pytest.mark.parametrize("to", [0, 5, -300_000], ids=["more", "after", "before"])
def test_bucket_above_a_block(ctx, to, threads):
    """One bucket of 210,000 tuples, the scan's last unit: it takes the device-wide sort, which has to see the mismatch."""
    data = _poly_c(3000)
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(31, st)
        job.partition(31, 1, threads, st, cnt.chunk_first_read, cnt.hist)
        want = job.labels()
        c = np.diff(cnt.hist.astype(np.int64))
        b = int(np.argmax(c))
        assert c[b] > 12_288 and b > 300_000
        c[b + to] += 1
        if to:
            c[b] -= 1
        bad = np.r_[0, np.cumsum(c)].astype(np.uint64)
        with pytest.raises(native.MetapartError) as e:
            job.partition(31, 1, threads, st, cnt.chunk_first_read, bad)
        assert code(e.value) == EFMT
        job.partition(31, 1, threads, st, cnt.chunk_first_read, cnt.hist)
        assert np.array_equal(job.labels(), want)


def _dip(h):  # one value below the one before
    b = int(np.searchsorted(h, h[-1] // 2)) + 50
    h[b] = h[b - 1] - 1


def _saw(h):  # every second one: a unit at most buckets, where the right prefix has a hundredth of them
    h[2001:900_001:2] += np.uint64(50_000)


def _past(h):  # a bucket that seems to hold a million tuples
    h[300_000] += np.uint64(1 << 20)


@pytest.mark.parametrize("fall", [_dip, _saw, _past], ids=["dip", "saw", "past"])
@pytest.mark.parametrize("n,k,scans,threads", [(600, 27, 1, 1), (60_000, 31, 1, 1), (60_000, 31, 1, 4), (60_000, 31, 2, 4)],
                         ids=["600", "60000", "60000-t4", "60000-s2"])
def test_falling_prefix(ctx, n, k, scans, threads, fall):
    """A prefix that somewhere falls.  (The planner may refuse the ranges that it finds in it.)"""
    data = synth.fastq_bytes(synth.workload("plain_large", n, seed=23))
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(k, st)
        job.partition(k, scans, threads, st, cnt.chunk_first_read, cnt.hist)
        want = job.labels()
        bad = cnt.hist.copy()
        fall(bad)
        with pytest.raises(native.MetapartError) as e:
            job.partition(k, scans, threads, st, cnt.chunk_first_read, bad)
        assert code(e.value) in (EFMT, EUNSUP)
        job.partition(k, scans, threads, st, cnt.chunk_first_read, cnt.hist)
        assert np.array_equal(job.labels(), want)
