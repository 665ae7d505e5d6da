"""Device memory of scans that are split together: the split tuples of all scans go back when a partition fails, and
when a later scan has to be sorted (a read that the scan before hooked below a component) and needs the room itself; a
request of the loop takes no more for them than was set aside for it.
"""
import threading

import numpy as np
import pytest

from metapart_gb300 import native, serve, synth

pytestmark = pytest.mark.gpu


def _starts(data, chunks=4):
    fno, ofs = native.fastq_index(chunks, [data])
    return native.chunk_starts_of(fno, ofs, [len(data)])


def test_failed_partition_keeps_no_split_tuples(built_gpu):
    data = synth.fastq_bytes(synth.workload("hotspot", 40_000, seed=31))
    st = _starts(data)
    with native.Context(0) as ctx, native.Job(ctx) as job:
        job.load(data)
        cnt = job.count(27, st)
        tuples = int(cnt.hist[-1])
        used = []
        for _ in range(3):
            job.set_wait_limits(union_retries=1)
            with pytest.raises(native.MetapartError, match="union-find"):
                job.partition(27, 2, 4, st, cnt.chunk_first_read, cnt.hist)
            used.append(ctx.hbm_in_use())
        assert used[2] - used[0] < 1 << 20 < 12 * tuples
        job.set_wait_limits()
        job.partition(27, 2, 4, st, cnt.chunk_first_read, cnt.hist)


def _hooked(n):
    """Two scans of n reads, the second after a BAD read was hooked in the first (bad_anchor_fastq's "two_scans", larger)."""
    L = 100
    reads = ["A" * (L - 1) + c for c in "CGTC"] + ["C" * L] * n + [("GC" * L)[:L]] * n
    return "".join(f"@b{i}\n{s}\n+\n{'I' * len(s)}\n" for i, s in enumerate(reads)).encode()


def test_sorted_scan_after_merged_ones_fits_where_it_did(built_gpu):
    """Every budget that holds the two scans one after another holds them when they may be split together."""
    data = _hooked(60_000)
    st = _starts(data)

    def run(budget, together):
        with native.Context(0, hbm_budget=budget) as ctx, native.Job(ctx) as job:
            job.load(data)
            cnt = job.count(27, st)
            total = int(cnt.hist[-1])
            job.set_scan_piece_tuples(total if together else total - 1)
            try:
                job.partition(27, 2, 1, st, cnt.chunk_first_read, cnt.hist)
            except native.MetapartError as e:
                assert "(-4)" in str(e)  # MP_ENOMEM
                return None
            assert job.scan_pieces == 2
            return job.labels()

    mb = 1 << 20
    lo, hi = 64, 2048  # does not fit, fits
    want = run(hi * mb, False)
    assert want is not None
    while hi - lo > 8:
        m = (lo + hi) // 2
        if run(m * mb, False) is None:
            lo = m
        else:
            hi = m
    for b in range(hi, hi + 320, 16):
        got = run(b * mb, True)
        assert got is not None, f"budget {b} MB (one after another: {hi} MB)"
        assert np.array_equal(got, want)


def test_request_stays_within_its_footprint(built_gpu):
    """A small k, long reads and three scans without a store: the scans split together would take more than the request's
    reservation, one after another they do not."""
    import torch
    spec = synth.workload("plain_large", 300_000, seed=33)
    spec.lengths = (250,)
    data = synth.fastq_to(spec, lambda n: (lambda t: (t, t.data_ptr()))(torch.empty(n, dtype=torch.uint8, pin_memory=True)))
    out = torch.empty(data.numel() + 64, dtype=torch.uint8, pin_memory=True)
    p = serve.RequestParams(k=11, num_scans=3, num_threads=4, num_chunks=8, read_store=0)
    with native.Context(0) as ctx, serve.Server(ctx, slots=1) as srv:
        ticket = srv.submit(data.data_ptr(), data.numel(), p, out.data_ptr(), out.numel())
        peak, done = [0], threading.Event()

        def watch():
            while not done.is_set():
                peak[0] = max(peak[0], ctx.hbm_in_use())

        w = threading.Thread(target=watch)
        w.start()
        try:
            r = srv.result(ticket)
        finally:
            done.set()
            w.join()
    assert r.status == 0, r.error
    assert data.numel() < peak[0] <= serve.footprint(data.data_ptr(), data.numel(), p)
