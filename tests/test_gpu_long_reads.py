"""Counting where a few reads are much longer than the rest (or all are): the histogram against counts made on the host, at
the lengths where reads change to a block of their own, and that one long read does not set the time of all.
"""
import numpy as np
import pytest

from metapart_gb300 import native, synth

pytestmark = pytest.mark.gpu

NB = 1 << 20


@pytest.fixture(scope="module")
def ctx(built_gpu):
    c = native.Context(0)
    yield c
    c.close()


def _counts(read, k):
    """Bucket counts of one read's canonical k-mers (A0 C1 G2 T3; no window with an N)."""
    code = np.array([{65: 0, 67: 1, 71: 2, 84: 3}.get(c, 0) for c in read], dtype=np.uint64)
    m = len(read) - k + 1
    if m < 2:  # (a read of k bases is not counted)
        return np.zeros(NB, np.int64)
    f, r = np.zeros(m, np.uint64), np.zeros(m, np.uint64)
    for i in range(k):
        f = (f << np.uint64(2)) | code[i:i + m]
        r |= (np.uint64(3) - code[i:i + m]) << np.uint64(2 * i)
    n = np.convolve(np.array([c == 78 for c in read], int), np.ones(k, int), "valid") == 0
    b = (np.minimum(f, r) >> np.uint64(2 * (k - 10)))[n]
    return np.bincount(b.astype(np.int64), minlength=NB)


def _fastq(reads):
    return b"".join(b"@r%d\n%s\n+\n%s\n" % (i, r, b"I" * len(r)) for i, r in enumerate(reads))


@pytest.mark.parametrize("store", ["fastq", "packed"])
@pytest.mark.parametrize("k", [11, 17, 31])
@pytest.mark.parametrize("lengths", [(1535, 1536), (1536, 1537), (100, 512, 513, 1537), (60, 4096), (4096, 4095, 600), (31, 32, 2049)],
                         ids=str)
def test_counts(ctx, lengths, k, store):
    rng = np.random.default_rng(sum(lengths) + k)
    reads = []
    for i in range(300):
        r = rng.choice(list(b"ACGT"), lengths[i % len(lengths)] if i % 7 == 0 or len(lengths) < 3 else lengths[0]).astype(np.uint8)
        r[rng.random(len(r)) < 0.003] = ord("N")
        reads.append(r.tobytes())
    data = _fastq(reads)
    with native.Job(ctx) as job:
        job.set_read_store(store)
        job.load(data)
        cnt = job.count(k, np.array([0, len(data)], np.uint64), want_chunk_counts=True)
    want = sum(_counts(r, k) for r in reads)
    assert np.array_equal(np.diff(cnt.hist.astype(np.int64)), want)
    assert np.array_equal(cnt.chunk_counts[0].astype(np.int64), want)


def test_one_long_read_does_not_set_the_time(ctx):
    short = synth.fastq_bytes(synth.workload("plain_small", 600_000, seed=2))
    long_ = b"@l\n" + b"ACGTTGCA" * 500 + b"\n+\n" + b"I" * 4000 + b"\n"
    t = []
    for data in (short, short + long_):
        with native.Job(ctx) as job:
            best = 1e9
            for _ in range(4):
                job.reset()
                job.load(data)
                job.count(27, np.array([0, len(data)], np.uint64))
                best = min(best, job.stage_ms()["count"])
            t.append(best)
    assert t[1] < 5 * t[0], t  # (8.5 with the tiles that the long read set)
