"""Budgets that a job fits with every allocation exact: what a job needs follows from its input, not from the blocks that
small allocations are cut from, nor from where the histogram's prefix is made.
"""
import numpy as np
import pytest

from metapart_gb300 import native, synth

pytestmark = pytest.mark.gpu

NB = 1 << 20


def _least(f, lo, hi):
    assert f(hi)
    while hi - lo > 16384:
        m = (lo + hi) // 2
        lo, hi = (lo, m) if f(m) else (m, hi)
    return hi


def _fits(data, budget, stage, k=27):
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    with native.Context(0, hbm_budget=budget) as c, native.Job(c) as j:
        try:
            j.load(data)
            if stage == "count":
                j.count(k, st)
        except native.MetapartError as e:
            assert "(-4)" in str(e)  # MP_ENOMEM
            return False
    return True


def test_load(built_gpu):
    """The bytes, the newlines' positions (8 bytes each, four a record) and the record table (20 a record)."""
    n = 20_000
    data = synth.fastq_bytes(synth.workload("plain_small", n, seed=3))
    least = _least(lambda b: _fits(data, b, "load"), 1 << 20, 64 << 20)
    assert least < len(data) + 52 * n + (256 << 10)


def test_count(built_gpu):
    """Beside what stays of the load (the bytes and the table), the counts of 2^20 buckets: the prefix is then the host's."""
    n = 20_000
    data = synth.fastq_bytes(synth.workload("plain_small", n, seed=3))
    least = _least(lambda b: _fits(data, b, "count"), 1 << 20, 64 << 20)
    assert least < len(data) + 20 * n + 8 * NB + (256 << 10)
    fno, ofs = native.fastq_index(4, [data])
    st = native.chunk_starts_of(fno, ofs, [len(data)])
    got = []
    for budget in (least, 0):
        with native.Context(0, hbm_budget=budget) as c, native.Job(c) as j:
            j.load(data)
            got.append(j.count(27, st).hist)
    assert np.array_equal(*got) and int(got[0][-1]) == n * 74
