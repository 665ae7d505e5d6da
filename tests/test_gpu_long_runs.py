"""Runs of one k-mer longer than a block (the oversized units), whose reads are all or nearly all BAD or whose k-mer is
zeroed or zero: the grouped scan against the sorted one, and that the unions do not look through such a run from each of its
stretches.

Reads that hold a 64-base adapter between random bases: the adapter's first and last 31-mers branch on one side, which makes
every such read BAD, so each of its inner k-mers has a long run of BAD reads.  A read of inner bases alone is not BAD and
joins its like, wherever they lie in the run.
"""
import numpy as np
import pytest

from metapart_gb300 import native
from test_gpu_group import _same

pytestmark = pytest.mark.gpu

ADAPTER = np.random.default_rng(8).choice(list(b"ACGT"), 64).astype(np.uint8)


@pytest.fixture(scope="module")
def ctx(built_gpu):
    c = native.Context(0)
    yield c
    c.close()


def _records(bases):
    """Equally long reads (an array of rows) as FASTQ bytes."""
    n, length = bases.shape
    a = np.empty((n, 9 + length + 3 + length + 1), np.uint8)
    a[:, 0] = ord("@")
    a[:, 1:8] = np.char.zfill(np.arange(n).astype("U7"), 7).astype("S7").view(np.uint8).reshape(n, 7)
    a[:, 8] = 10
    a[:, 9:9 + length] = bases
    a[:, 9 + length:12 + length] = np.frombuffer(b"\n+\n", np.uint8)
    a[:, 12 + length:12 + 2 * length] = ord("I")
    a[:, -1] = 10
    return a.tobytes()


def _adapters(n, frac, length=110, seed=3):
    rng = np.random.default_rng(seed)
    b = rng.choice(list(b"ACGT"), (n, length)).astype(np.uint8)
    b[rng.random(n) < frac, 20:84] = ADAPTER
    return b


def _starts_of(data, chunks):
    fno, ofs = native.fastq_index(chunks, [data])
    return native.chunk_starts_of(fno, ofs, [len(data)])


def _inner(m):
    return _records(np.repeat(ADAPTER[None, 5:60], m, 0)) if m else b""


@pytest.mark.parametrize("inner", [0, 2, 6])
@pytest.mark.parametrize("scans", [1, 2])
def test_reads_all_bad(ctx, inner, scans):
    b = _records(_adapters(30_000, 0.9))
    half = len(b) // 2
    data = b[:half] + _inner(inner // 2) + b[half:] + _inner(inner - inner // 2)
    _same(ctx, data, 31, 4, scans, 2)
    if inner:
        starts = _starts_of(data, 4)
        with native.Job(ctx) as job:
            job.load(data)
            cnt = job.count(31, starts)
            job.partition(31, scans, 2, starts, cnt.chunk_first_read, cnt.hist)
            lab = job.labels()
        at = list(range(15_000, 15_000 + inner // 2)) + list(range(len(lab) - (inner - inner // 2), len(lab)))
        assert len(set(lab[at].tolist())) == 1


@pytest.mark.parametrize("base", [b"A", b"C"])
def test_one_letter_reads(ctx, base):
    """The zero k-mer (no read joins) and the run of one k-mer (all join), beside others."""
    b = _adapters(4_000, 0.5)
    b[1::2] = base[0]
    b[0:40:2, 60:] = base[0]
    _same(ctx, _records(b), 31, 4, 1, 2)


def test_unions_pass_by_bad_reads(ctx):
    """The unions of 33 runs of a million BAD reads take less time than half of their judgement (looked through from every
    stretch, they took longer than it)."""
    data = _records(_adapters(1_500_000, 0.9))
    starts = _starts_of(data, 4)
    with native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(31, starts)
        best = None
        for _ in range(3):
            job.partition(31, 1, 2, starts, cnt.chunk_first_read, cnt.hist)
            t = job.stage_ms()
            best = t if best is None or t["union_find"] < best["union_find"] else best
    assert best["union_find"] < 0.5 * best["filter"], best
